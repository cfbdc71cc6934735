"""The attach's host loops over the mesh stay a function of their own: inlined into
the attach they cost it 1.4 times its time."""
import shutil
import subprocess

import pytest

from gdon3d_b200 import capi


@pytest.mark.skipif(shutil.which("nm") is None, reason="needs nm")
def test_neighbour_rows_are_built_out_of_line():
    names = subprocess.run(["nm", "-C", capi.LIB_PATH], capture_output=True, text=True, check=True).stdout
    assert " t build_neighbours(" in names
