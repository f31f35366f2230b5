"""The shared-memory layout of the pressure solve along grid lines, checked on the CPU.

The CTAs of a cluster store into one another's shared memory (the neighbours' values and mbarriers, the
sums of a reduction, the flag that asks for a sweep to be repeated) at their own offsets, while each
CTA has its own number of rows with a well's fill.  The layout header the kernel uses is compiled
here with g++.
"""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def layout_lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("layout") / "pencil_layout_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", out,
                    os.path.join(HERE, "native", "pencil_layout_host.cpp")], check=True)
    return C.CDLL(out)


@pytest.mark.parametrize("value_bytes", [4, 8])
@pytest.mark.parametrize("nx,nz,cols,cs", [(40, 5, 4, 2), (21, 5, 5, 4), (45, 7, 4, 16), (127, 40, 7, 16)])
def test_places_other_ctas_store_to_do_not_depend_on_the_wells(layout_lib, value_bytes, nx, nz, cols, cs):
    def places(wells, entries):
        out = (C.c_int64 * 5)()
        layout_lib.rfh_pencil_remote_places(value_bytes, nx, nz, cols, cs, 8, 128, wells, entries, out)
        return list(out)
    base = places(0, 0)
    for wells, entries in ((1, 7), (nz, 4 * nz * nz), (2 * nz, 9 * nz * nz)):
        here = places(wells, entries)
        assert here[:4] == base[:4]
        assert here[4] > max(here[:4])
