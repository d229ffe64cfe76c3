"""The two-row marches at the sizes where they can go wrong, against the FP64
oracle: columns one node under, at and over the 32 lanes and the 8 rows (and
one row of a thread's two), z depths from one plane, one-node axes, several z
chunks, body force, 16-bit storage.

Bounds (FP32): a step rounds each moment in a few operations of relative error
eps = 6e-8; the sums carry deviations of O(u), so the second moments (O(u^2))
are off by some eps / u.  With u ~ 0.02 and 6 steps: 64 eps on rho and u,
64 eps / 0.02 on the second moments.  16-bit storage rounds every moment each
step to 11 (8) bits: 6 steps of half an ulp on u, 4 times that on the others.
"""
import numpy as np
import pytest

import mrlbm
import parity_util as pu

pytestmark = pytest.mark.gpu
EPS = 6e-8
STEPS = 6
SHAPES = [(31, 7, 1), (32, 8, 3), (33, 9, 2), (1, 12, 10), (12, 1, 5), (9, 5, 1), (64, 16, 33), (65, 17, 40), (2, 2, 2),
          (40, 23, 67)]


def flow(shape, seed):
    rng = np.random.default_rng(seed)
    return [1 + 0.001 * rng.standard_normal(shape), *(0.02 * rng.standard_normal((3,) + shape))]


def errors(d, chunk=0, nt=None):
    dom = mrlbm.Domain(d)
    if nt is not None:
        dom.set_node_types(nt)
    shape = (d.nz, d.ny, d.nx)
    dom.init_flow(*flow(shape, d.nx * 7 + d.ny * 3 + d.nz))
    if chunk:
        dom.set_z_chunk(chunk)
    orc = pu.oracle_for(d, nt)
    orc.set_moments(pu.gpu_to_oracle_layout(dom.moments()))
    dom.step(STEPS)
    orc.step(STEPS)
    fluid = None if nt is None else np.asarray(nt) != mrlbm.NODE_SOLID
    res = pu.compare(dom.moments(), orc.moments(), fluid=fluid)
    dom.close()
    return max(res[k][0] for k in range(4)), max(res[k][0] for k in range(4, 10))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("force", [False, True])
def test_d3q27_bulk(shape, force):
    f = (2e-5, -1e-5, 3e-5) if force else (0.0, 0.0, 0.0)
    d = mrlbm.make_desc(*shape, lattice=mrlbm.D3Q27, tau=0.56, force=f)
    for chunk in (0, 1, min(3, shape[2])):
        low, second = errors(d, chunk)
        assert low < 64 * EPS and second < 64 * EPS / 0.02, (shape, chunk, low, second)


@pytest.mark.parametrize("storage,ulp", [(mrlbm.F16, 2.0 ** -11), (mrlbm.BF16, 2.0 ** -8), (mrlbm.F16U, 2.0 ** -20)])
@pytest.mark.parametrize("shape", [(33, 9, 2), (64, 16, 33)])
def test_d3q27_16bit(shape, storage, ulp):
    d = mrlbm.make_desc(*shape, lattice=mrlbm.D3Q27, storage=storage, tau=0.6)
    low, second = errors(d)
    # split storage keeps the second moments (and the little they give u) in one fp16 word
    assert low < STEPS * max(ulp, 2.0 ** -14 if storage == mrlbm.F16U else 0.0), low
    assert second < 4 * STEPS * max(ulp, 2.0 ** -11), second
