"""ORACLE — test infrastructure only.

Location of the mounted reference sources, for the recipes that read them in
place (oracle/Makefile `make ref`, the golden-fixture scripts under
tests/golden/) and the tests that replay the reference's own files. The
environment variable SUNDOG_REFERENCE names the reference checkout; without
it the recipes look at the one mount point this project's build machines
use. Nothing here is needed where the reference is absent: the prebuilt
oracle/_ref libraries travel with the repository, and code that needs the
sources checks for None.
"""

import os

_DEFAULT_MOUNT = "/root/reference"


def reference_root():
    """The reference checkout's root directory, or None when it is absent (an
    empty mount point counts as absent: there is nothing in it to compile)."""
    r = os.environ.get("SUNDOG_REFERENCE") or _DEFAULT_MOUNT
    return r if os.path.isfile(os.path.join(r, "src", "capi_scene.cpp")) else None
