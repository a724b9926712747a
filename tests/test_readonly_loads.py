"""The step's kernels are launched overlapped, so a kernel may start while the
one before it still writes the state and the packed records.  Read-only loads
(__ldg, ld.global.nc) are for data that no kernel writes meanwhile: in the
kernels' sources they take mesh arrays and the work list only."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nextgen_b200", "csrc")

# a mesh array, a halo list, or (in Rows and ROWS_START) the row streams that
# ROWS_START is given, themselves mesh arrays
MESH = re.compile(r"(reinterpret_cast<const double2\*>\()?\(?(m\.\w+|halo\b|ROWS_OF\b|src\b|idx\b|eidx\b)")


def code(name):
    s = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", s)


def test_read_only_loads_take_mesh_data():
    text = code("cgx.cu") + code("cgx_mixed.cuh")
    loads = re.findall(r"__ldg\(([^;\n]*)", text)
    assert len(loads) >= 30
    assert [a for a in loads if not MESH.match(a)] == []
    assert ".nc." not in text
    assert "eidx = m.lidx" in text
    rows = re.findall(r"ROWS_START\(([^\n]*?)\)\n", text)
    used = [r for r in rows if "ROWS_OF" not in r]
    assert len(used) == 16
    assert all(re.match(r"m\.\w+, [xyz], m\.\w+, m\.\w+, ", r) for r in used), used
