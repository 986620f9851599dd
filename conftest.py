"""Environment of the test run.

The shim's tests look for the reference's headers in $PIC3D_REFERENCE/include;
with the variable unset that is ./include, this repository's own headers, taken
for the reference's.  Where the variable is unset and no reference build exists
it names a directory that does not exist, and the tests that need the reference
are skipped, as they say.
"""
import os

REPO = os.path.dirname(os.path.abspath(__file__))
if not os.path.isdir(os.path.join(REPO, "oracle", "_ref")):
    os.environ.setdefault("PIC3D_REFERENCE", os.path.join(REPO, "no_reference"))
