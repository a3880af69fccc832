"""The marching sweeps at the edges of their strips (26 output columns a warp,
four warps a block, 4 to 128 output rows) and the two forms of the remap, bit
for bit against the oracle: one step on smooth and on rough fields, whose
slopes switch every limiter and the positivity filter."""
import numpy as np
import pytest

from atmdyn import ic, Dycore
import pyoracle

pytestmark = pytest.mark.gpu

FIELDS = (('dp', pyoracle.DP), ('pt', pyoracle.PT), ('ud', pyoracle.UD), ('vd', pyoracle.VD))


def rough(nx, ny, nlay, seed):
    """Log-normal thickness and potential temperature (ratios of neighbours up
    to about a hundred), winds of both signs and some exact ties."""
    st = ic.bubble_case(nx, ny, nlay, 50e3, 50e3, seed=seed)
    rng = np.random.default_rng(seed)
    st.dp = st.dp * np.exp(rng.normal(0, 1.2, st.dp.shape))
    st.pt = st.pt * np.exp(rng.normal(0, 1.2, st.pt.shape))
    st.u = np.round(rng.normal(0, 15.0, st.u.shape), 0)
    st.v = rng.normal(0, 15.0, st.v.shape)
    return st


# nx, ny around the strip widths (104 columns a block, halo rows and columns
# 2-3 wide), the smallest domain, and one tall enough for 128-row strips
SIZES = [(7, 7, 3), (26, 33, 5), (27, 8, 4), (100, 9, 3), (105, 131, 3), (416, 270, 24)]


@pytest.mark.parametrize('nx,ny,nlay', SIZES)
@pytest.mark.parametrize('fields', ['smooth', 'rough'])
def test_step_bit_exact(nx, ny, nlay, fields):
    st = rough(nx, ny, nlay, nx) if fields == 'rough' else ic.jet_case(nx, ny, nlay, 400e3, 400e3, width=900e3, seed=ny)
    dt = 20.0 if fields == 'rough' else 60.0
    g, o = Dycore(st), pyoracle.OracleModel(st, threads=8)
    for a in (g, o):
        a.cgrid_step(dt / 2)
        a.cgrid_halo()
    for name, f in (('dpc', pyoracle.DPC), ('ptc', pyoracle.PTC), ('uc', pyoracle.UC), ('vc', pyoracle.VC)):
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    for a in (g, o):
        a.dgrid_step(dt)
        a.dgrid_halo()
    for name, f in FIELDS:
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    g.close()


@pytest.mark.parametrize('nx,ny,nlay', [(60, 9, 3), (140, 41, 3), (235, 18, 3)])
def test_narrow_blocks_bit_exact(nx, ny, nlay):
    """Widths of 3, 6 and 10 strips, whose blocks hold three, three and two."""
    test_step_bit_exact(nx, ny, nlay, 'rough')


@pytest.mark.parametrize('nx,ny,nlay', [(9, 8, 3), (23, 17, 32), (40, 33, 33), (20, 18, 65), (12, 11, 128),
                                        (300, 270, 8)])
@pytest.mark.parametrize('fields', ['smooth', 'rough', 'crossed'])
def test_remap_bit_exact(nx, ny, nlay, fields):
    """The remap alone, in its shared-level form (few columns; the three layer
    ranges) and with one thread a column (the last size), with its layer-pair
    trace; crossed: some columns whose interfaces are not monotone, which take
    the all-pairs search."""
    st = ic.jet_case(nx, ny, nlay, 400e3, 400e3, width=900e3, seed=ny)
    rng = np.random.default_rng(nlay)
    if fields != 'smooth':
        st.dp = st.dp * np.exp(rng.normal(0, 0.7, st.dp.shape))
        st.pt = st.pt * np.exp(rng.normal(0, 0.1, st.pt.shape))
        st.u = st.u + rng.normal(0, 15.0, st.u.shape)
        st.v = st.v + rng.normal(0, 15.0, st.v.shape)
    if fields == 'crossed':
        st.dp[1] = np.where(rng.random((ny, nx)) < 0.03, -0.2 * st.dp[1], st.dp[1])
    g, o = Dycore(st), pyoracle.OracleModel(st, threads=8)
    small = nx < 100
    if small:
        trace_o = o.enable_trace()
        trace_g, fallback = g.remap_trace()
    g.remap()
    o.remap()
    for name, f in FIELDS:
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    if small:
        np.testing.assert_array_equal(trace_g, trace_o)
        # (the face interpolation crosses some coordinates of the rough fields too)
        assert fallback.value > 0 if fields == 'crossed' else fields == 'rough' or fallback.value == 0
    g.close()


@pytest.mark.parametrize('nlay', [21, 30, 45, 46, 47, 61, 62, 63])
def test_layer_counts_near_shared_limit(nlay):
    """Layer counts whose column arrays fill the 48 KB that a block may take
    without opting in, with and without room for the kernels' own variables:
    the remap and its reverse launch, first thing in the process for some."""
    st = ic.jet_case(9, 8, nlay, 400e3, 400e3, width=900e3, seed=nlay)
    g, o = Dycore(st), pyoracle.OracleModel(st, threads=8)
    g.adj_enable()
    g.adj_remap()
    g.remap()
    o.remap()
    for name, f in FIELDS:
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    g.close()


@pytest.mark.parametrize('nx,ny,nlay', [(7, 8, 3), (19, 9, 33), (10, 9, 128), (300, 250, 4)])
def test_heating_bit_exact(nx, ny, nlay):
    """A step with the heating term of a radiative net flux, and the finite
    check over the same shapes."""
    import torch
    st = ic.jet_case(nx, ny, nlay, 400e3, 400e3, width=900e3, seed=ny)
    nf = np.random.default_rng(nx).normal(0, 150.0, (nlay + 1, ny + 14, nx + 14))
    g, o = Dycore(st), pyoracle.OracleModel(st, threads=8)
    for a in (g, o):
        a.set_net_flux(nf)
        a.cgrid_step(15.0)
        a.cgrid_halo()
        a.dgrid_step(30.0)
        a.dgrid_halo()
    for name, f in FIELDS:
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    pt = g.get('pt')
    assert g.check_stability()
    for bad in (np.nan, np.inf):
        for at in ((0, 0, 0), (nlay - 1, ny - 1, nx - 1)):
            p = pt.copy()
            p[at] = bad
            g.upload_device('pt', torch.from_numpy(p).cuda())
            assert not g.check_stability()
    g.close()


@pytest.mark.parametrize('nx,ny,nlay', [(257, 255, 3), (254, 241, 97), (249, 247, 64), (243, 240, 97)])
def test_column_pass_both_sides_of_the_limit(nx, ny, nlay):
    """Column passes of (nx + 4)(ny + 4) columns just above and just below the
    limits up to which their levels are shared."""
    test_step_bit_exact(nx, ny, nlay, 'smooth')


@pytest.mark.parametrize('nx,ny,nlay', [(147, 143, 3), (300, 290, 10), (270, 263, 97)])
def test_heating_thread_a_column_bit_exact(nx, ny, nlay):
    """The heating term of domains of many columns."""
    test_heating_bit_exact(nx, ny, nlay)


# columns beyond which a thread has a column of its own, in each of the kernels'
# layer ranges (the limits depend on the layers)
@pytest.mark.parametrize('nx,ny,nlay', [(161, 152, 3), (211, 200, 8), (290, 270, 33), (203, 190, 65), (140, 137, 128)])
@pytest.mark.parametrize('fields', ['smooth', 'crossed'])
def test_remap_thread_a_column_bit_exact(nx, ny, nlay, fields):
    """The remap of domains of many columns with its layer-pair trace."""
    st = ic.jet_case(nx, ny, nlay, 400e3, 400e3, width=900e3, seed=ny)
    rng = np.random.default_rng(nlay)
    st.dp = st.dp * np.exp(rng.normal(0, 0.2, st.dp.shape))
    st.u = st.u + rng.normal(0, 15.0, st.u.shape)
    st.v = st.v + rng.normal(0, 15.0, st.v.shape)
    if fields == 'crossed':
        st.dp[1] = np.where(rng.random((ny, nx)) < 0.01, -0.2 * st.dp[1], st.dp[1])
    g, o = Dycore(st), pyoracle.OracleModel(st, threads=8)
    trace_o = o.enable_trace()
    trace_g, fallback = g.remap_trace()
    g.remap()
    o.remap()
    for name, f in FIELDS:
        np.testing.assert_array_equal(g.get(name, halo=True), o.get(f, halo=True), err_msg=name)
    np.testing.assert_array_equal(trace_g, trace_o)
    if fields == 'crossed':
        assert fallback.value > 0
    g.close()


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('nlay', [10, 70])
def test_tiled_domain_same_bits(precision, nlay):
    """A domain of copies of a smaller one: each copy is the smaller domain's
    step, heating and remap bit for bit, although the larger one's columns are
    too many for the forms that share a column's levels.  (The remap after the
    halo fill: within a step it reads winds of the old halo, as the reference
    does, which the larger domain's inner copies do not have.)"""
    nx, ny, my, mx = 70, 65, 5, 4
    st = ic.jet_case(nx, ny, nlay, 400e3, 400e3, width=900e3, seed=3)
    rng = np.random.default_rng(nlay)
    st.dp = st.dp * np.exp(rng.normal(0, 0.05, st.dp.shape))
    st.u = st.u + rng.normal(0, 10.0, st.u.shape)
    st.v = st.v + rng.normal(0, 10.0, st.v.shape)
    nf = rng.normal(0, 150.0, (nlay + 1, ny, nx))
    big = ic.jet_case(nx * mx, ny * my, nlay, 400e3, 400e3, width=900e3, seed=3)
    for name in ('dp', 'pt', 'u', 'v', 'gzs'):
        a = getattr(st, name)
        setattr(big, name, np.tile(a, (1,) * (a.ndim - 2) + (my, mx)))
    out = []
    for s, flux in ((st, nf), (big, np.tile(nf, (1, my, mx)))):
        g = Dycore(s, precision)
        g.set_net_flux(np.pad(flux, ((0, 0), (7, 7), (7, 7)), mode='wrap'))
        for _ in range(2):
            assert g.step(20.0, remap=False, check_stable=True)
            g.remap()
            g.dgrid_halo()
        out.append({name: g.get(name) for name, _ in FIELDS})
        g.close()
    for name, _ in FIELDS:
        np.testing.assert_array_equal(out[1][name], np.tile(out[0][name], (1, my, mx)), err_msg=name)
