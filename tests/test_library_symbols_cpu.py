"""The library shares no statics with another build of itself in the process:
the loader merges symbols of the unique type across libraries, and with them the
tables a kernel takes."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG


def test_no_process_unique_symbols():
    lib = os.path.join(PKG, "lib", "libsipg_gb300.so")
    if not os.path.exists(lib) or not shutil.which("nm"):
        pytest.skip("library not built, or no nm")
    out = subprocess.run(["nm", "-D", "--defined-only", lib], capture_output=True, text=True, check=True).stdout
    unique = [line for line in out.splitlines() if line.split()[1:2] == ["u"]]
    assert not unique, unique[:3]
