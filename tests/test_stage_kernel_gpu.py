"""The TMA stage kernel at the sizes where its tiles, tile sets and coefficients
change, and the host-buffer RHS at the edges of its staging pieces."""
import numpy as np
import pytest

import oracle
from oracle import Geom, Params

from test_parity_gpu import parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import granite_b200
    return granite_b200


def _state(o, g, seed):
    u = o.init_brill_lindquist(g, [1.0], [[0.12, -0.1, 0.05]], r_floor=0.5 * g.dx[0])
    u = oracle.add_noise(u, 1e-10, seed)
    u[19:22] += 0.05 * oracle.hash_noise((3,) + g.shape[1:], seed)  # shifts of both signs
    return u


def _run(gb, geoms, states, precision, batched=True, chi=0.0, cfg=None, steps=2):
    ev = gb.Evolver(gb.CCZ4Params())
    if cfg is not None:
        ev.force_stage_config(cfg)
    ev.set_batching(batched)
    blocks = []
    for i, (g, u) in enumerate(zip(geoms, states)):
        b = gb.GridBlock(i, 0, g.n, g.lo, g.hi)
        b.array[...] = u
        ev.add_block(b)
        blocks.append(b)
    if chi:
        ev.set_fp64_chi_threshold(chi)
    ev.commit()
    ev.upload()
    dt = 0.25 * geoms[0].dx[0]
    for _ in range(steps):
        ev.rk3_step(0, dt, precision, gb.BC_REFERENCE)
    ev.download()
    ev.close()
    return [b.array.copy() for b in blocks], dt


# one tile and less, exact tiles, remainders of 8 (both tile sets) and of 2 in x,
# partial tiles in y and z, more tiles than warpgroups
@pytest.mark.parametrize("n", [(16, 4, 4), (16, 4, 5), (18, 6, 4), (24, 4, 4), (24, 12, 6), (40, 18, 10), (48, 48, 48)])
@pytest.mark.parametrize("cfg", [None, 0, 12])
def test_fp64_steps_match_the_oracle(gb, oracle_lib, n, cfg):
    g = Geom(n, tuple(-0.125 * a for a in n), tuple(0.125 * a for a in n))
    u = _state(oracle_lib, g, 3)
    (out,), dt = _run(gb, [g], [u], gb.PRECISION_FP64, cfg=cfg)
    # 2 steps of rounding-level differences (20 steps are held to 1e-10 elsewhere)
    parity(out, oracle_lib.rk3_steps(Params(), g, u, dt, 2), rtol=1e-11, what=f"{n}, cfg {cfg}")


@pytest.mark.parametrize("precision,chi", [(0, 0.0), (1, 0.0), (1, 0.5), (1, 0.999999)])
def test_blocks_of_different_spacing_share_a_launch(gb, oracle_lib, precision, chi):
    """The kernel reads the coefficients of a level whose blocks differ in them from
    the descriptors, one launch for the level or one per block: the same kernel,
    the same bits. A block alone has its coefficients in the kernel arguments. The
    two kernels may contract the algebra differently: a few units in the last
    place of the RHS per stage in FP64 (6 stages, below 1e-13), of FP32 in the
    mixed form."""
    geoms = [Geom((24, 20, 16), (-3.0, -2.5, -2.0), (3.0, 2.5, 2.0)),
             Geom((32, 16, 18), (4.0, 4.0, 4.0), (13.6, 9.2, 9.7)),
             Geom((18, 22, 14), (-9.0, -9.0, -9.0), (-4.5, -3.5, -5.5))]
    states = [_state(oracle_lib, g, 10 + i) for i, g in enumerate(geoms)]
    a, _ = _run(gb, geoms, states, precision, True, chi)
    b, _ = _run(gb, geoms, states, precision, False, chi)
    for i in range(len(geoms)):
        assert np.array_equal(a[i], b[i]), f"block {i}: batched and block by block"
    # (the first block: the step length is its own)
    (alone,), _ = _run(gb, geoms[:1], states[:1], precision, True, chi)
    parity(a[0], alone, rtol=1e-13 if precision == 0 else 1e-6, what="the first block alone")


# 24^3 cells of 8 bytes are less than a staging piece; 64 x 40: a field is several
# pieces with a ragged last one; x of 300: rows that do not divide a piece
@pytest.mark.parametrize("n", [(16, 16, 16), (64, 40, 33), (300, 12, 11)])
def test_host_rhs_writes_the_interior_only(gb, oracle_lib, n):
    g = Geom(n, tuple(-0.125 * a for a in n), tuple(0.125 * a for a in n))
    u = _state(oracle_lib, g, 5)
    b, rhs = gb.GridBlock(0, 0, g.n, g.lo, g.hi), gb.GridBlock(1, 0, g.n, g.lo, g.hi)
    b.array[...] = u
    rhs.array[...] = np.arange(rhs.array.size, dtype=np.float64).reshape(rhs.array.shape)
    before = rhs.array.copy()
    op = gb.CCZ4Evolution(gb.CCZ4Params())
    op.computeRHSVacuum(b, rhs)
    inner = np.zeros(rhs.array.shape, bool)
    inner[rhs.interior()] = True
    assert np.array_equal(rhs.array[~inner], before[~inner])
    once = rhs.array.copy()
    op.computeRHSVacuum(b, rhs)  # the pieces are handed out again
    assert np.array_equal(rhs.array, once)
    it = rhs.interior()
    parity(rhs.array[it], oracle_lib.rhs(Params(), g, u)[it], rtol=1e-12, what=f"{n}")
