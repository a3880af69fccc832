"""Adjoint of the FP64 step on the GPU against the oracle's tangent-linear model.

Dot-product tests: for random tangents v of a stage's inputs (the CPU
tangent-linear oracle, branches frozen at the FP64 trajectory) and random
adjoints w of its outputs (the CUDA adjoint kernels), <w, J v> and
<J^T w, v> agree to 1e-12 relative.  The base state is a bubble with
noise on every field, so that no limiter sits exactly on a tie (a tie is a
kink where the one-sided derivatives differ).
"""
import copy

import numpy as np
import pytest

from atmdyn import ic, Dycore
import pyoracle

pytestmark = pytest.mark.gpu

H = 7
TOL = 1e-12
NAMES = ('dp', 'pt', 'ud', 'vd')
STATE = {'dp': pyoracle.DP, 'pt': pyoracle.PT, 'ud': pyoracle.UD, 'vd': pyoracle.VD}
CGRID = {'dpc': pyoracle.DPC, 'ptc': pyoracle.PTC, 'uc': pyoracle.UC, 'vc': pyoracle.VC}
SCALE = {'dp': 10.0, 'pt': 0.01, 'ud': 0.5, 'vd': 0.5, 'dpc': 10.0, 'ptc': 0.01, 'uc': 0.5, 'vc': 0.5}


def generic_state(nx=40, ny=24, nlay=6, seed=0):
    st = ic.bubble_case(nx, ny, nlay, 200e3, 200e3, radius=800e3, u0=12.0)
    rng = np.random.default_rng(seed)
    st.v = st.v + 2.0
    st.dp = st.dp + rng.normal(0, 5.0, st.dp.shape)
    st.pt = st.pt * (1 + rng.normal(0, 1e-3, st.pt.shape))
    st.u = st.u + rng.normal(0, 0.5, st.u.shape)
    st.v = st.v + rng.normal(0, 0.5, st.v.shape)
    return st


def padded_shape(st):
    return (st.nlay, st.ny + 2 * H, st.nx + 2 * H)


def rand(rng, st, name):
    return rng.normal(0, SCALE[name], padded_shape(st))


def mask(st, r):
    m = np.zeros(padded_shape(st))
    m[:, H - r:H + st.ny + r, H - r:H + st.nx + r] = 1.
    return m


def rel(a, b):
    return abs(a - b) / max(abs(a), abs(b), 1e-300)


def tlm_from_gpu(g, st, tangents):
    """A tangent-linear oracle whose state values are the GPU's padded fields."""
    t = pyoracle.TLMModel(st)
    for n in NAMES:
        t.set(STATE[n], g.get(n, halo=True), tangents.get(n), halo=True)
    return t


def test_cgrid_step_dot_product():
    st = generic_state()
    rng = np.random.default_rng(1)
    g = Dycore(st)
    g.adj_enable()
    v = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, v)
    t.cgrid_step(st.dt / 2)
    w = {n: rand(rng, st, n) * mask(st, 2 if n in ('dpc', 'ptc') else 0) for n in CGRID}
    lhs = sum(np.sum(w[n] * t.get(CGRID[n], halo=True)[1]) for n in CGRID)
    for n in CGRID:
        g.adj_set('in', n, w[n])
    g.adj_cgrid_step(st.dt / 2)
    rhs = sum(np.sum(v[n] * g.adj_get('in', n)) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


def test_dgrid_step_dot_product():
    st = generic_state(seed=2)
    rng = np.random.default_rng(3)
    g = Dycore(st)
    g.adj_enable()
    vs = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, vs)
    t.cgrid_step(st.dt / 2)
    t.cgrid_halo()
    vc = {n: rand(rng, st, n) for n in CGRID}
    for n in CGRID:
        t.set(CGRID[n], t.get(CGRID[n], halo=True)[0], vc[n], halo=True)
    t.dgrid_step(st.dt)
    w = {n: rand(rng, st, n) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n], halo=True)[1]) for n in NAMES)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_dgrid_step(st.dt)
    rhs = sum(np.sum(vs[n] * g.adj_get('in', n)) for n in NAMES)
    rhs += sum(np.sum(vc[n] * g.adj_get('in', n)) for n in CGRID)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


@pytest.mark.parametrize('nx,ny,nlay', [(7, 7, 3), (27, 9, 3), (31, 40, 4), (113, 13, 3), (121, 131, 3)])
def test_strip_edges_dot_product(nx, ny, nlay):
    """The C and D step together at the edges of the reverse kernels' strips
    (26 to 30 columns a warp, four warps a block, 4 to 128 rows), on log-normal
    thickness and potential temperature, whose slopes reach the positivity
    filter and both sides of every limiter."""
    st = generic_state(nx, ny, nlay, seed=nx)
    rng = np.random.default_rng(ny)
    st.dp = st.dp * np.exp(rng.normal(0, 1.0, st.dp.shape))
    st.pt = st.pt * np.exp(rng.normal(0, 1.0, st.pt.shape))
    st.u = st.u + rng.normal(0, 15.0, st.u.shape)
    st.v = st.v + rng.normal(0, 15.0, st.v.shape)
    dt = 30.0
    g = Dycore(st)
    g.adj_enable()
    vs = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, vs)
    t.cgrid_step(dt / 2)
    t.cgrid_halo()
    t.dgrid_step(dt)
    w = {n: rand(rng, st, n) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n], halo=True)[1]) for n in NAMES)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_dgrid_step(dt)
    g.adj_cgrid_halo()
    g.adj_cgrid_step(dt / 2)
    rhs = sum(np.sum(vs[n] * g.adj_get('in', n)) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


def test_remap_dot_product():
    st = generic_state(seed=4)
    rng = np.random.default_rng(5)
    g = Dycore(st)
    g.adj_enable()
    g.cgrid_step(st.dt / 2)
    g.cgrid_halo()
    g.dgrid_step(st.dt)  # the pre-remap state, with last step's ring on the winds
    v = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, v)
    t.remap()
    w = {n: rand(rng, st, n) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n], halo=True)[1]) for n in NAMES)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_remap()
    rhs = sum(np.sum(v[n] * g.adj_get('in', n)) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


def test_remap_dot_product_non_monotone_columns():
    """Columns whose source pressure is not monotone (one layer of negative
    thickness) take the all-pairs path of the remap and of its adjoint."""
    st = generic_state(seed=6)
    for j, i in ((3, 5), (10, 20), (17, 31)):
        st.dp[2, j, i] = -0.3 * st.dp[2, j, i]
    rng = np.random.default_rng(7)
    g = Dycore(st)
    g.adj_enable()
    v = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, v)
    t.remap()
    w = {n: rand(rng, st, n) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n], halo=True)[1]) for n in NAMES)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_remap()
    rhs = sum(np.sum(v[n] * g.adj_get('in', n)) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


def test_halo_dot_products():
    st = generic_state(seed=6)
    rng = np.random.default_rng(7)
    g = Dycore(st)
    g.adj_enable()
    v = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, v)
    t.dgrid_halo()
    w = {n: rand(rng, st, n) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n], halo=True)[1]) for n in NAMES)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_halo('out')
    rhs = sum(np.sum(v[n] * g.adj_get('out', n)) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)
    # the C-grid fields
    t.cgrid_step(st.dt / 2)
    vc = {n: rand(rng, st, n) for n in CGRID}
    for n in CGRID:
        t.set(CGRID[n], t.get(CGRID[n], halo=True)[0], vc[n], halo=True)
    t.cgrid_halo()
    wc = {n: rand(rng, st, n) for n in CGRID}
    lhs = sum(np.sum(wc[n] * t.get(CGRID[n], halo=True)[1]) for n in CGRID)
    for n in CGRID:
        g.adj_set('in', n, wc[n])
    g.adj_cgrid_halo()
    rhs = sum(np.sum(vc[n] * g.adj_get('in', n)) for n in CGRID)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


@pytest.mark.parametrize('remap_every', [2, 100])
def test_three_steps_dot_product(remap_every):
    """Three whole steps (C, halo, D, [remap], halo) through atm_adj_step."""
    st = generic_state(32, 24, 6, seed=8)
    rng = np.random.default_rng(9)
    nsteps = 3
    v = {n: rng.normal(0, SCALE[n], (st.nlay, st.ny, st.nx)) for n in NAMES}
    t = pyoracle.TLMModel(st, v)
    for s in range(nsteps):
        t.cgrid_step(st.dt / 2)
        t.cgrid_halo()
        t.dgrid_step(st.dt)
        if (s + 1) % remap_every == 0:
            t.remap()
        t.dgrid_halo()
    w = {n: rng.normal(0, SCALE[n], (st.nlay, st.ny, st.nx)) for n in NAMES}
    lhs = sum(np.sum(w[n] * t.get(STATE[n])[1]) for n in NAMES)
    lam = {n: np.pad(w[n], ((0, 0), (H, H), (H, H))) for n in NAMES}
    for s in reversed(range(nsteps)):
        g = Dycore(st)
        for q in range(s):
            g.step(st.dt, remap=(q + 1) % remap_every == 0, check_stable=False)
        g.adj_enable()
        for n in NAMES:
            g.adj_set('out', n, lam[n])
        g.adj_step(st.dt, remap=(s + 1) % remap_every == 0)
        lam = {n: g.adj_get('out', n) for n in NAMES}
        if s == 0:
            g.adj_halo('out')
            lam = {n: g.adj_get('out', n, halo=False) for n in NAMES}
        g.close()
    rhs = sum(np.sum(v[n] * lam[n]) for n in NAMES)
    assert rel(lhs, rhs) <= TOL, (lhs, rhs)


@pytest.mark.parametrize('nx,ny,nlay', [(9, 8, 3), (13, 9, 20), (20, 17, 32), (9, 8, 33), (11, 8, 64), (8, 7, 65),
                                        (7, 8, 128), (250, 240, 54)])
def test_layer_counts_dot_product(nx, ny, nlay):
    """The columns' and the remap's reverse over the ranges of their column
    arrays (up to 32, 64 and 128 layers), on columns that differ enough for
    layers to overlap several targets and for all pair cases.  The bound is on
    the sum of the products' magnitudes: the reverse rounds each term a few
    hundred times at most."""
    st = generic_state(nx, ny, nlay, seed=nlay)
    rng = np.random.default_rng(nx)
    st.dp = st.dp * np.exp(rng.normal(0, 0.3, st.dp.shape))
    g = Dycore(st)
    g.adj_enable()
    v = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, v)
    dt = 10.0
    for a in (t, g):
        a.cgrid_step(dt / 2)
        a.cgrid_halo()
        a.dgrid_step(dt)
        a.remap()
    w = {n: rand(rng, st, n) for n in NAMES}
    terms = [w[n] * t.get(STATE[n], halo=True)[1] for n in NAMES]
    g.close()
    g = Dycore(st)
    g.adj_enable()
    g.cgrid_step(dt / 2)
    g.cgrid_halo()
    g.dgrid_step(dt)
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_remap()
    back = {n: g.adj_get('in', n) for n in NAMES}
    g.close()
    # the step before the remap, from its initial state
    g = Dycore(st)
    g.adj_enable()
    for n in NAMES:
        g.adj_set('out', n, back[n])
    g.adj_dgrid_step(dt)
    g.adj_cgrid_halo()
    g.adj_cgrid_step(dt / 2)
    rhs = sum(np.sum(v[n] * g.adj_get('in', n)) for n in NAMES)
    lhs, scale = sum(np.sum(x) for x in terms), sum(np.sum(np.abs(x)) for x in terms)
    assert abs(lhs - rhs) <= TOL * scale, (lhs, rhs, scale)
    g.close()


@pytest.mark.parametrize('nx,ny,nlay', [(190, 151, 3), (313, 287, 9), (310, 306, 12), (312, 305, 33),
                                        (231, 224, 70), (162, 157, 113)])
def test_many_columns_dot_product(nx, ny, nlay):
    """Domains of more columns than the limits beyond which a thread has a column
    of its own, of few layers (both reverses of the remap, that of the columns) and of more."""
    test_layer_counts_dot_product(nx, ny, nlay)


def test_tall_domain_dot_product():
    """The reverse of a step of a domain of more rows than a grid holds rows of
    blocks (65535).  The bound is on the sum of the products' magnitudes."""
    nx, ny, nlay = 7, 65600, 3
    st = generic_state(nx, ny, nlay, seed=9)
    rng = np.random.default_rng(10)
    dt = 30.0
    g = Dycore(st)
    g.adj_enable()
    vs = {n: rand(rng, st, n) for n in NAMES}
    t = tlm_from_gpu(g, st, vs)
    t.cgrid_step(dt / 2)
    t.cgrid_halo()
    t.dgrid_step(dt)
    w = {n: rand(rng, st, n) for n in NAMES}
    terms = [w[n] * t.get(STATE[n], halo=True)[1] for n in NAMES]
    for n in NAMES:
        g.adj_set('out', n, w[n])
    g.adj_dgrid_step(dt)
    g.adj_cgrid_halo()
    g.adj_cgrid_step(dt / 2)
    rhs = sum(np.sum(vs[n] * g.adj_get('in', n)) for n in NAMES)
    lhs, scale = sum(np.sum(x) for x in terms), sum(np.sum(np.abs(x)) for x in terms)
    assert abs(lhs - rhs) <= TOL * scale, (lhs, rhs, scale)
    g.close()


def test_launch_count():
    """Every kernel of the reverse is counted, the clears and the copies of a
    tape among them."""
    import torch
    g = Dycore(generic_state(20, 17, 5, seed=3))
    g.adj_enable()
    tape = torch.empty(g.tape_bytes() // 8, dtype=torch.float64, device='cuda')

    def count(f):
        n = g.launch_count()
        f()
        return g.launch_count() - n
    assert count(g.adj_zero) == 2
    # C step recomputed 3, column 1, momentum 4 (clear, x, y, rest), column 1, mass 2
    assert count(lambda: g.adj_cgrid_step(10.0)) == 11
    # winds recomputed 1, clear 1, energy 1, winds 1, ring 1
    assert count(g.adj_remap) == 5
    # C step 3, halo 1, copy 1, D step 5, copy 1, halo 1
    assert count(lambda: g.step_tape(20.0, False, tape.data_ptr())) == 12
    # halo 1, clear 1, D step 2 + 3 + 2 + 1, halo 1, C step 8
    assert count(lambda: g.adj_step_tape(20.0, False, tape.data_ptr())) == 19
    # ... with the forward step recomputed (3 + 1 + 5)
    assert count(lambda: g.adj_step(20.0, remap=False)) == 28
    # ... and the remap's reverse with its clear
    assert count(lambda: g.adj_step(20.0, remap=True)) == 34
    g.close()


def test_tape_alignment():
    """The tape is written alike on 16-byte and on 8-byte boundaries."""
    import torch
    st = generic_state(9, 8, 5, seed=3)
    tapes = []
    for shift in (0, 1):
        g = Dycore(st)
        n = g.tape_bytes() // 8
        buf = torch.full((n + 2,), 7.0, dtype=torch.float64, device='cuda')
        g.step_tape(st.dt, True, buf.data_ptr() + 8 * shift)
        torch.cuda.synchronize()
        tapes.append(buf[shift:shift + n].cpu().numpy())
        assert buf[shift + n].item() == 7.0 and (shift == 0 or buf[0].item() == 7.0)
        g.close()
    np.testing.assert_array_equal(tapes[0], tapes[1])
