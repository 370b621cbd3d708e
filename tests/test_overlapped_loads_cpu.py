"""Kernels that are launched while the one before them still runs read its
results with ordinary loads.  The read-only path is defined only for data that
nobody writes during the kernel's life, and such a load may be moved above the
wait for the kernel before; only tables that no kernel writes may take it.
(Read from the source: on the device a wrong load gives right results most of
the time.)"""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "eisenjoch_b200" / "csrc"
# twiddles, spectral weights and wave numbers: uploaded with the bin grid
TABLES = ("tb.tw", "tb.tq", "a.wx", "a.wy", "a.gx2", "a.gy2")


def test_read_only_loads_are_of_tables():
    files = [f for f in sorted(CSRC.glob("*.cu*")) if "griddepcontrol.wait" in f.read_text()]
    assert files
    for f in files:
        text = re.sub(r"//[^\n]*", "", f.read_text())
        assert "ld.global.nc" not in text, f.name
        for arg in re.findall(r"__ldg\(\s*([^;]*)", text):
            assert arg.startswith(TABLES), (f.name, arg[:60])
