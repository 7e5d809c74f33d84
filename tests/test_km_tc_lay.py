"""The shapes that the small-k tensor-core assignment takes and the shared
memory it lays out for them (yael_gb300/csrc/km_tc_lay.h), on the host."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LIMIT = 227 * 1024


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("kmtc") / "libkmtcshim.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-o", out,
                    os.path.join(HERE, "km_tc_shim.cpp")], check=True)
    lib = ctypes.CDLL(out)
    lib.shim_tc_total.restype = ctypes.c_long
    return lib


def test_shapes_and_layouts(shim):
    """Every whole-float4 d up to 192 with every k up to 256, up to 256 with k up
    to 128, and no other; for each, with and without sums, two stages at least
    and a pair list of 32 at least within the limit, and nothing left out that
    would fit beside those."""
    out = (ctypes.c_long * 6)()
    for d in range(1, 261):
        for k in range(1, 260):
            ok = d % 4 == 0 and k <= 256 and (d <= 192 or (d <= 256 and k <= 128))
            assert bool(shim.shim_tc_shape_ok(d, k)) == ok, (d, k)
            if not ok:
                continue
            csm_wanted = int((k + 31) // 32 * 32 * d * 4 <= 32 * 1024)
            for sums in (0, int(k * d * 8 <= 48 * 1024)):
                shim.shim_tc_lay(d, k, sums, out)
                total, S, fuse, csm, xs, pairs = out

                def over(*form):
                    return shim.shim_tc_total(d, k, *form) > LIMIT
                assert total <= LIMIT and 2 <= S <= 6 and pairs in (32, 64), (d, k)
                assert S == 6 or over(S + 1, fuse, csm, xs, pairs), (d, k)
                assert pairs == 64 or over(2, fuse, csm, xs, 64), (d, k)
                assert xs or over(2, sums, csm_wanted, 1, 32), (d, k)
                assert csm == csm_wanted or over(2, sums, 1, 0, 32), (d, k)
                assert fuse == sums or over(2, 1, 0, 0, 32), (d, k)
