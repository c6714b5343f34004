"""The step kernels' dispatch and tile edges against the oracle, bit for bit
(GPU): rows one past a tile, a last y tile of one quad, shells that end inside
a quad, a chunk per plane and one chunk, segments of deferred cells that
overflow (the step is then re-run), and amplitudes that send the reference
arithmetic's divisions by the spacing through each of its three forms.  Every
result is compared by its bits, so there is no tolerance to choose; the adjoint
on shells that end inside a quad is held to the cosines of test_adjoint.py (the
delta gradient, whose signal is S with its threshold, to 0.99)."""
import numpy as np
import pytest

import qp3d
import synthetic
from oracle import oracle as O
from helpers import bits_equal
from test_gpu_parity import _live_pml_mask

pytestmark = pytest.mark.gpu

NT = 8


@pytest.fixture
def sctx(ctx):
    yield ctx
    ctx.tune(arith=1, tile_x=0, chunks=0, spec_delta_ppm=10000, threshold_mode=1)


def _check(ctx, shot, u_prev, u_cur, pml_state, arith):
    ctx.tune(arith=arith)
    ctx.load(shot)
    ctx.write_state(0, u_prev, u_cur, pml_state)
    ctx.advance(shot.nt)
    rec, mx = ctx.record(), ctx.uxyzmax()
    g_prev, g_cur, g_pml = ctx.read_state()
    prob = shot.to_oracle(O)
    st = O.State(prob)
    st.u1[:], st.u2[:], st.u3[:], st.pml[:] = u_prev, u_cur, u_cur, pml_state
    orec, omx, st = O.run(O.MIRROR if arith else O.REF32, prob, state=st)
    assert bits_equal(mx, omx)
    assert bits_equal(rec, orec)
    assert bits_equal(g_cur, st.u2) and bits_equal(g_prev, st.u1)
    live = _live_pml_mask(shot.nx, shot.ny, shot.nz, shot.pml)
    assert bits_equal(g_pml[live], st.pml[live])


@pytest.mark.parametrize("arith", [1, 0])
@pytest.mark.parametrize("hx,hy,nz0,pml,tile_x,chunks", [
    (31, 23, 14, 6, 0, 0),      # 43 x 35 x 26: 33 updated rows, shells of 6
    (18, 19, 17, 7, 32, 1),     # 32 x 33 x 31: one quad, of one cell, in the last y tile
    (29, 53, 13, 5, 16, 13),    # 39 x 63 x 23: one plane a chunk, shells of 5
    (40, 25, 22, 0, 11, 2),     # 40 x 25 x 22: no shell
    (16, 90, 16, 9, 24, 3),     # 34 x 108 x 34: three quads in the last y tile
    (37, 26, 15, 6, 0, 0)])     # 49 x 38 x 27: two
def test_tile_edges(sctx, hx, hy, nz0, pml, tile_x, chunks, arith):
    shot = synthetic.small_case(hx=hx, hy=hy, nz0=nz0, pml=pml, nt=NT, seed=61,
                                src=(hx // 2, hy // 2, nz0 // 2))
    sctx.tune(tile_x=tile_x, chunks=chunks)
    _check(sctx, shot, *synthetic.random_state(shot, seed=61), arith)


@pytest.mark.parametrize("scale", [2.0 ** -120, 2.0 ** -75, 2.0 ** 33])
def test_reference_divisions_at_any_amplitude(sctx, scale):
    """Windows below, across and above the range in which a quotient by the
    spacing is taken without scaling."""
    shot = synthetic.small_case(hx=22, hy=26, nz0=18, pml=6, nt=NT, seed=62)
    shot.wavelet[:] *= np.float32(scale)
    state = [np.asarray(a * np.float32(scale)) for a in synthetic.random_state(shot, seed=62)]
    _check(sctx, shot, *state, 0)


def overflow_case():
    """A ramp whose slope is the threshold's over most of the grid, under a blob
    that sets the maximum: most cells of a column are deferred."""
    shot = synthetic.small_case(hx=60, hy=40, nz0=30, pml=6, nt=NT, seed=63)
    nz, nx, ny = shot.nz, shot.nx, shot.ny
    z, x, y = np.meshgrid(np.arange(nz), np.arange(nx), np.arange(ny), indexing="ij")
    r2 = (z - nz / 2) ** 2 + (x - 16) ** 2 + (y - 16) ** 2
    blob = np.exp(-r2 / (2 * 3.0 ** 2))                 # slope 0.202 a cell at its steepest
    u = (blob + 0.00202 * (x - nx / 2)).astype(np.float32).ravel()
    return shot, u, np.zeros_like(O.State(shot.to_oracle(O)).pml)


@pytest.mark.parametrize("arith", [1, 0])
def test_overflowing_segments_rerun_the_step(sctx, arith):
    """Against the steps with the maximum known beforehand: the state here fills
    the never-updated outer cells, which the oracle's copies and the library's
    rotation hand on differently."""
    shot, u, pml_state = overflow_case()
    out = []
    for mode in (0, 1):
        sctx.tune(arith=arith, threshold_mode=mode, spec_delta_ppm=250000)
        sctx.load(shot)
        sctx.write_state(0, u, u, pml_state)
        sctx.advance(shot.nt)
        out.append((sctx.record(), sctx.uxyzmax()) + tuple(sctx.read_state()[:2]))
        redo, _ = sctx.stats()
    assert redo.any()
    for a, b in zip(*out):
        assert bits_equal(a, b)


@pytest.mark.parametrize("hy,pml", [(19, 5), (18, 6), (21, 7)])
def test_adjoint_of_shells_that_end_inside_a_quad(hy, pml):
    shot = synthetic.small_case(hx=21, hy=hy, nz0=17, pml=pml, nt=80, seed=64, fm=30.0)
    rng = np.random.default_rng(64)
    with qp3d.Context(0) as c:
        d_obs = c.forward(shot)
        d_obs = (d_obs * (1 + 0.1 * rng.standard_normal(d_obs.shape))).astype(np.float32)
        _, g = c.adjoint(shot, d_obs)
    adj = O.Adjoint(shot.to_oracle(O), live=True).freeze()
    rec, hist = adj.forward(want_hist=True)
    g64 = adj.backward(hist, rec - d_obs.astype(np.float64))
    for a, b, least in zip(g, g64, (0.999, 0.999, 0.99)):
        assert float(np.dot(a, b) / (np.linalg.norm(a) * np.linalg.norm(b))) >= least
