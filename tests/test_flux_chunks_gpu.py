"""Chunks of planes of the collocated flux kernel (csrc/flux_ring.cuh, k_flux_coll.cu): where a
plane has nearly a wave of tiles, a chunk must not outgrow the table of plane constants, beyond
which the same plane took other roundings.

On an equidistant mesh (spacing 3/64, exact in both precisions) a velocity that repeats every other plane has an
explicit term that does, bit for bit, whatever chunk a plane is in.  The tiles are 32 x 8 nodes
in FP64 and 32 x 16 in the mixed form, a wave 296 and 444 CTAs: 256 tiles (one chunk), and 144
(two) of a long column."""
import numpy as np
import pytest

from cases import COLLOC, make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,NX,NY,NZ", [(0, 512, 128, 150), (0, 192, 192, 300), (1, 1024, 128, 139)])
def test_planes_of_a_period_are_equal(precision, NX, NY, NZ):
    import turbchannel_b200 as tb

    prod, _, _ = make_case(COLLOC, NX, NY, NZ, precision=precision)
    zz = np.arange(NZ) * (3.0 / 64.0)
    prod["area"] = prod["hx"] * NX * prod["hy"] * NY * (zz[-1] - zz[0])
    S = tb.Solver(prod, zz)
    v = np.random.default_rng(2).standard_normal((2, NY * NX, 3))
    v = np.tile(v, ((NZ + 1) // 2, 1, 1))[:NZ].copy()
    v[0] = v[-1] = 0.0
    f = np.asarray(S.ExplicitTerm(v.reshape(-1, 3))).reshape(NZ, -1)
    S.close()
    for z in range(4, NZ - 2):
        assert np.array_equal(f[z], f[z - 2]), z
