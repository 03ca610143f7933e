"""The launch record of the FP64 sum names the CTAs per SM of the instance that ran: at least the four
that the 16- and 32-column instances are built for, three of the 64-column one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_ctas_per_sm_of_the_fp64_instances(bie, rng):
    itf = bie.single_dielectric_box3d(1.2, 0.8, 0.6, 4, 0.2, 4.0, 1.0)
    op = bie.lhs_dielectric_box3d(itf)
    ctas = {}
    for k in (8, 16, 32, 64):
        op @ np.asfortranarray(rng.standard_normal((itf.n, k)))
        ctas[k] = bie.tuned_launch(op, "fp64", k)["ctas_per_sm"]
    assert ctas[8] >= 3 and ctas[16] >= 4 and ctas[32] >= 4 and ctas[64] == 3, ctas
