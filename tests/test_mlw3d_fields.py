"""The table of fields of the marching 3-D steps (kVar in mlw3d_march.cuh): a difference
that a column retains belongs to one variable, and so to one of the two threads of its
cell; a variable without a flux in a direction names none.  CPU only."""
import re
from pathlib import Path

from utrip_gb300 import build


def table():
    text = (Path(build.CSRC) / "mlw3d_march.cuh").read_text()
    names = re.search(r"struct VarFields \{\s*signed char ([^;]*);", text).group(1)
    body = re.search(r"kVar\[8\] = \{(.*?)\};", text, re.S).group(1)
    keys = [k.strip() for k in names.split(",")]
    return [dict(zip(keys, (w.strip() for w in row.split(","))))
            for row in re.findall(r"\{([^{}]*)\}", body)]


def test_retained_differences_have_one_owner():
    rows = table()
    assert len(rows) == 8
    for flux, corner, kept in (("fx", "kx", "rx"), ("fy", "ky", "ry")):
        slots = [r[kept] for r in rows if r[flux] != "-1"]
        assert sorted(map(int, slots)) == list(range(7))
        for r in rows:
            assert (r[flux] == "-1") == (r[corner] == "-1") == (r[kept] == "-1"), r
