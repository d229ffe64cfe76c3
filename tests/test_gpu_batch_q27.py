"""D3Q27 batches: members that the sums march, the populations march and the
wall solve take, chained in the same persistent CTAs, equal the same domains
stepped alone bit for bit (and the forced ones the FP64 oracle).  Forced members
without walls do so where they are in the sums march, FP32 ones always."""
import numpy as np
import pytest

import mrlbm
import parity_util as pu

pytestmark = pytest.mark.gpu
STEPS = 21   # odd: one replayed graph of 16 launches, then single ones


def bulk(nx, ny, nz, storage, force=(0.0, 0.0, 0.0)):
    return mrlbm.make_desc(nx, ny, nz, lattice=27, storage=storage, tau=0.6, force=force), None


def cavity(nx, ny, nz, storage):
    d = mrlbm.lid_cavity_desc(nx, re=60.0, lid_u=0.05, lattice=27, storage=storage, ny=ny, nz=nz)
    return d, mrlbm.lid_cavity_node_types(nx, ny, nz, 1)


def duct(n, storage, rheology, seed):
    rng = np.random.default_rng(seed)
    solid = np.zeros((n, n, n), dtype=np.uint8)
    solid[:, 1:-1, 1:-1] = rng.random((n, n - 2, n - 2)) < 0.05
    d = mrlbm.make_desc(n, n, n, lattice=27, storage=storage, periodic=(0, 0, 1), tau=0.8, force=(0, 0, 2e-5),
                        rheology=rheology, nnf_n=0.8)
    return d, mrlbm.voxel_node_types(solid, (0, 0, 1))


def start(dom, d, nt):
    rng = np.random.default_rng(d.nx * 7 + d.ny * 3 + d.nz)
    shape = (d.nz, d.ny, d.nx)
    if nt is not None:
        dom.set_node_types(nt)
    dom.init_flow(1 + 0.001 * rng.standard_normal(shape), *(0.02 * rng.standard_normal((3,) + shape)))


def members(storage):
    """Ragged sizes around the 32 lanes and the 8 and 14 rows, z depths over
    and under the batch's chunk of 32, each march next to the others."""
    return [bulk(33, 9, 40, storage), cavity(31, 15, 34, storage), bulk(40, 23, 7, storage, (2e-5, -1e-5, 3e-5)),
            duct(18, storage, mrlbm.NEWTONIAN, 1), bulk(64, 14, 33, storage), duct(20, storage, mrlbm.POWERLAW, 2),
            bulk(1, 12, 10, storage), bulk(32, 28, 2, storage, (1e-5, 0.0, 0.0)), cavity(33, 8, 5, storage),
            bulk(512, 312, 2, storage), bulk(520, 330, 2, storage, (0.0, 1e-5, 0.0)), bulk(2, 2, 2, storage)]


@pytest.mark.parametrize("rows", [8, 14])
@pytest.mark.parametrize("storage", [mrlbm.F32, mrlbm.F16, mrlbm.F16U])
def test_members_equal_alone(storage, rows):
    b = mrlbm.Batch(mrlbm.D3Q27, storage)
    b.set_rows(rows)
    mem = []
    for d, nt in members(storage):
        m = b.add(d)
        start(m, d, nt)
        mem.append(m)
    b.step(STEPS)
    b.synchronize()
    for (d, nt), m in zip(members(storage), mem):
        dom = mrlbm.Domain(d)
        start(dom, d, nt)
        dom.step(STEPS)
        dom.synchronize()
        got, want, name = m.moments(), dom.moments(), "%d x %d x %d" % (d.nx, d.ny, d.nz)
        if storage != mrlbm.F32 and nt is None and any(d.force) and d.nx < 500:
            # the walls' kernel in the batch, the bulk one alone: the same
            # populations, products and sums contracted differently, so a
            # stored word differs by its rounding, a step at a time
            assert np.max(np.abs(got - want)) <= STEPS * 2.0 ** -11 * np.max(np.abs(want)), name
        else:
            np.testing.assert_array_equal(got, want, name)
        dom.close()
    b.close()


@pytest.mark.parametrize("rows", [8, 14])
def test_forced_members_against_the_oracle(rows):
    """FP32, 6 steps; the bounds of test_gpu_row_march (sums of deviations:
    64 eps on rho and u, that over u = 0.02 on the second moments)."""
    b = mrlbm.Batch(mrlbm.D3Q27, mrlbm.F32)
    b.set_rows(rows)
    cases = [bulk(33, 9, 40, mrlbm.F32, (2e-5, -1e-5, 3e-5)), bulk(40, 23, 7, mrlbm.F32), bulk(32, 28, 2, mrlbm.F32, (1e-5, 0, 0))]
    mem, orc = [], []
    for d, nt in cases:
        m = b.add(d)
        start(m, d, nt)
        o = pu.oracle_for(d)
        o.set_moments(pu.gpu_to_oracle_layout(m.moments()))
        mem.append(m)
        orc.append(o)
    b.step(6)
    for m, o in zip(mem, orc):
        o.step(6)
        res = pu.compare(m.moments(), o.moments())
        low, second = max(res[k][0] for k in range(4)), max(res[k][0] for k in range(4, 10))
        assert low < 64 * 6e-8 and second < 64 * 6e-8 / 0.02, (low, second)
    b.close()
