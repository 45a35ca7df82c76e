"""How the cooperative Krylov loops lay a system over the SMs, checked without a GPU."""
import numpy as np
import pytest

from platoanalyze_b200 import capi

WARPS = {3: 16, 1: 32}  # warps of a CTA by unknowns per row


def split(nslices, width, nb, sms, may_cluster):
    out = np.zeros(6, np.int32)
    slots = 32 * width * nslices
    rc = capi.lib.plato_test_pcg_split(nslices, slots, nb, sms, int(may_cluster), out.ctypes.data_as(capi.i32p))
    assert rc == capi.OK
    return dict(zip(("grid", "per_cta", "parts", "turns", "in_smem", "top"), out.tolist()))


@pytest.mark.parametrize("sms", [148, 20, 3])
@pytest.mark.parametrize("nb", [3, 1])
def test_leaders_stay_inside_the_partial_sums(nb, sms):
    """Whatever the number of slices, every slice of a CTA has a group of whole warps, and no leader reads
    beyond the CTA's 32 * warps partial sums, also where the warps do not divide among the slices."""
    warps, turns, odd = WARPS[nb], 1 if nb == 3 else 2, 0
    for n in list(range(1, 1200)) + [148 * warps * turns - 1, 148 * warps * turns]:
        for width in (2, 15, 40):
            for may_cluster in (False, True):
                s = split(n, width, nb, sms, may_cluster)
                assert 1 <= s["grid"] <= max(sms, 16) and s["grid"] * s["per_cta"] >= n
                groups = warps // s["parts"]
                assert groups * s["turns"] >= s["per_cta"]
                assert s["top"] < 32 * warps, (n, width, may_cluster, s)
                odd += warps % s["parts"] != 0
    assert odd > 0  # the case with warps left over is among them


def test_split_rejects_bad_input():
    out = np.zeros(6, np.int32).ctypes.data_as(capi.i32p)
    for args in ((0, 32, 3, 148), (1, 0, 3, 148), (1, 32, 2, 148), (1, 32, 3, 0)):
        assert capi.lib.plato_test_pcg_split(*args, 1, out) == capi.BAD_INPUT
