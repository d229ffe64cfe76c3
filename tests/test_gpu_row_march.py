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
WALL_LOW, WALL_SECOND = 2e-5, 3e-4   # whole populations: eps / u^2 on the second moments, as in test_gpu_parity
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
@pytest.mark.parametrize("shape", [(33, 9, 2), (512, 120, 2), (512, 128, 2), (515, 130, 3)])
def test_d3q27_16bit(shape, storage, ulp):
    """16-bit boxes of few and of 256 columns of 32 x 8 nodes (the line from
    which they take the sums march: test_16bit_one_step)."""
    d = mrlbm.make_desc(*shape, lattice=mrlbm.D3Q27, storage=storage, tau=0.6)
    low, second = errors(d)
    # split storage keeps the second moments (and the little they give u) in one fp16 word
    assert low < STEPS * max(ulp, 2.0 ** -14 if storage == mrlbm.F16U else 0.0), low
    assert second < 4 * STEPS * max(ulp, 2.0 ** -11), second


# unit roundoff of a stored word; velocity of the split storage: two words
UNIT = {mrlbm.F32: 2.0 ** -24, mrlbm.F16: 2.0 ** -11, mrlbm.BF16: 2.0 ** -8, mrlbm.F16U: 2.0 ** -11}


def one_step(d, seed, dev):
    """|error| after one step over its bound, the largest of each moment: the
    start is read back as stored, so a moment is off by the rounding of its
    own new word, unit * |moment|, and by FP32 sums of whole populations, 64 eps
    (times the stored scaling 3, 4.5 or 9).  Density deviations of `dev` are
    well over both."""
    shape = (d.nz, d.ny, d.nx)
    rng = np.random.default_rng(seed)
    dom = mrlbm.Domain(d)
    dom.init_flow(1 + dev * rng.standard_normal(shape), *(0.02 * rng.standard_normal((3,) + shape)))
    orc = pu.oracle_for(d)
    orc.set_moments(pu.gpu_to_oracle_layout(dom.moments()))
    dom.step(1)
    orc.step(1)
    got, want = pu.gpu_to_oracle_layout(dom.moments()), np.asarray(orc.moments(), dtype=np.float64)
    dom.close()
    out = []
    for k in range(10):
        unit = 2.0 ** -22 if d.storage == mrlbm.F16U and 1 <= k <= 3 else UNIT[d.storage]
        scale = 1.0 if k == 0 else 3.0 if k <= 3 else 9.0
        # 64 eps: the sums; the smallest words of FP16 (2^-24 over the storage scale of 8 at least)
        bound = unit * np.abs(want[..., k]) * (1 + 1e-3) + 64 * EPS * scale
        out.append(float(np.max(np.abs(got[..., k] - want[..., k]) / bound)))
    assert np.sqrt(np.mean(want[..., 0] ** 2)) > 0.5 * dev   # the deviations are there to be seen
    return out


@pytest.mark.parametrize("force", [False, True])
@pytest.mark.parametrize("storage", [mrlbm.F16, mrlbm.BF16, mrlbm.F16U])
@pytest.mark.parametrize("shape", [(33, 9, 2), (512, 304, 2), (512, 312, 2), (520, 330, 3)])
def test_16bit_one_step(shape, storage, force):
    """608, 624 and 714 columns of 32 x 8 nodes: both sides of the 1.4 waves of
    CTAs from which 16-bit moments take the sums march."""
    f = (2e-4, -1e-4, 3e-4) if force else (0.0, 0.0, 0.0)
    d = mrlbm.make_desc(*shape, lattice=mrlbm.D3Q27, storage=storage, tau=0.6, force=f)
    over = one_step(d, 3, 0.02)
    assert max(over) < 1.0, over


@pytest.mark.parametrize("force", [False, True])
@pytest.mark.parametrize("storage", [mrlbm.F32, mrlbm.F16, mrlbm.BF16])
@pytest.mark.parametrize("nz", [2660, 2700])   # as in test_d3q19_dense
def test_d3q19_dense_one_step(nz, storage, force):
    f = (2e-4, -1e-4, 3e-4) if force else (0.0, 0.0, 0.0)
    d = mrlbm.make_desc(33, 9, nz, lattice=mrlbm.D3Q19, storage=storage, tau=0.6, force=f)
    over = one_step(d, 4, 0.02)
    assert max(over) < 1.0, over


@pytest.mark.parametrize("shape,planes", [((160, 160, 160), 20), ((96, 300, 120), 20), ((224, 224, 224), 32),
                                          ((203, 173, 121), 25), ((340, 340, 24), 24)])
def test_d3q19_dense_chunks(shape, planes):
    """Not the one wave of long chunks, nor a few waves of them (40, 40, 112
    planes here once)."""
    dom = mrlbm.Domain(mrlbm.make_desc(*shape, lattice=mrlbm.D3Q19, tau=0.6))
    assert dom.z_chunk() == planes
    dom.close()


@pytest.mark.parametrize("nz", [2660, 2700])   # 4 columns: under and over 24 planes a CTA's place (10,656)
def test_d3q19_dense(nz):
    """The three-CTA shape of the D3Q19 bulk step, against the oracle, and bit
    for bit against the batch kernel (which has one shape)."""
    nx, ny = 33, 9
    d = mrlbm.make_desc(nx, ny, nz, lattice=mrlbm.D3Q19, tau=0.56)
    low, second = errors(d)
    assert low < WALL_LOW and second < WALL_SECOND, (low, second)
    dom, b = mrlbm.Domain(d), mrlbm.Batch(mrlbm.D3Q19, mrlbm.F32)
    m = b.add(d)
    f = flow((nz, ny, nx), 5)
    dom.init_flow(*f)
    m.init_flow(*f)
    dom.step(STEPS)
    b.step(STEPS)
    assert np.array_equal(dom.moments(), m.moments())
    b.close()
    dom.close()


# ---- walls that take the total sums (x and y faces) and the class table's order



def wall_errors(d, nt):
    low, second = errors(d, 0, nt)
    return low, second


@pytest.mark.parametrize("shape", [(33, 9, 5), (32, 8, 4), (5, 40, 6), (31, 7, 3)])
def test_d3q27_cavity(shape):
    nx, ny, nz = shape
    d = mrlbm.lid_cavity_desc(nx, re=20.0, lid_u=0.05, lattice=mrlbm.D3Q27, ny=ny, nz=nz)
    low, second = wall_errors(d, mrlbm.lid_cavity_node_types(nx, ny, nz, 1))
    assert low < WALL_LOW and second < WALL_SECOND, (low, second)


@pytest.mark.parametrize("storage,tol", [(mrlbm.F16, 2.0 ** -11), (mrlbm.BF16, 2.0 ** -8), (mrlbm.F16U, 2.0 ** -11)])
def test_d3q27_cavity_16bit(storage, tol):
    """The ghost shell's moments are subtracted as the storage rounds them."""
    nx, ny, nz = 33, 17, 9
    d = mrlbm.lid_cavity_desc(nx, re=20.0, lid_u=0.05, lattice=mrlbm.D3Q27, storage=storage, ny=ny, nz=nz)
    low, second = wall_errors(d, mrlbm.lid_cavity_node_types(nx, ny, nz, 1))
    assert low < 4 * STEPS * tol and second < 16 * STEPS * tol, (low, second)


@pytest.mark.parametrize("lattice", [mrlbm.D3Q19, mrlbm.D3Q27])
def test_inner_plane_typed_like_the_face(lattice):
    """The same node type on the x face (sources outside) and on an inner
    plane (fluid sources): only the face may take the total sums."""
    nx, ny, nz = 20, 10, 6
    nt = np.zeros((nz, ny, nx), dtype=np.uint32)
    nt[:, :, 0] = mrlbm.WEST
    nt[:, :, 11] = mrlbm.WEST
    nt[:, :, -1] = mrlbm.EAST
    d = mrlbm.make_desc(nx, ny, nz, lattice=lattice, periodic=(0, 1, 1), tau=0.7)
    low, second = wall_errors(d, nt)
    assert low < WALL_LOW and second < WALL_SECOND, (low, second)


@pytest.mark.parametrize("lattice", [mrlbm.D3Q19, mrlbm.D3Q27])
@pytest.mark.parametrize("rheology", [mrlbm.NEWTONIAN, mrlbm.POWERLAW])
@pytest.mark.parametrize("fill", [0.02, 0.3])
def test_scattered_obstacles(lattice, rheology, fill):
    """Few and (nearly) all of the 254 masks: the table in order of use, staged
    and past the staged classes."""
    nx, ny, nz = 34, 17, 12
    rng = np.random.default_rng(3)
    solid = np.zeros((nz, ny, nx), dtype=np.uint8)
    solid[:, 1:-1, 1:-1] = rng.random((nz, ny - 2, nx - 2)) < fill
    nt = mrlbm.voxel_node_types(solid, (0, 0, 1))
    d = mrlbm.make_desc(nx, ny, nz, lattice=lattice, periodic=(0, 0, 1), tau=0.8, force=(0, 0, 2e-5), rheology=rheology,
                        nnf_n=0.9)
    low, second = wall_errors(d, nt)
    assert low < 2 * WALL_LOW and second < 2 * WALL_SECOND, (low, second)


@pytest.mark.parametrize("shape,planes", [((32, 32, 32), 1), ((512, 8, 8), 1), ((40, 40, 40), 1), ((48, 48, 48), 2),
                                          ((128, 128, 128), 13), ((99, 62, 139), 11), ((256, 256, 256), 32),
                                          ((160, 160, 160), 23)])
def test_sums_march_chunks(shape, planes):
    """Few tiles: the shortest chunk of one wave, one plane if that fits; the
    planes evenly spread over the chunks (128: ten of 13, not nine of 14 and
    one of 2)."""
    dom = mrlbm.Domain(mrlbm.make_desc(*shape, lattice=mrlbm.D3Q27, tau=0.6))
    assert dom.z_chunk() == planes
    dom.close()
