"""The kernels that pass over whole rows (device uploads and downloads, adjoint
sets and gets, the finite check) at each width of their thread groups and where
a row is cut into pieces: values, halos and the smallest bad value anywhere."""
import numpy as np
import pytest

from atmdyn import ic, Dycore

pytestmark = pytest.mark.gpu

H = 7
# widths of 7 to 64 threads a group and of several rounds, with and without the
# halo, and wide domains of few rows (several pieces a row, the last one short)
SIZES = [(7, 7, 3), (16, 40, 3), (19, 9, 4), (50, 8, 3), (70, 11, 5), (129, 8, 3), (300, 300, 8), (1031, 7, 3),
         (4099, 7, 3)]


@pytest.mark.parametrize('nx,ny,nlay', SIZES)
def test_fields_in_and_out(nx, ny, nlay):
    import torch
    st = ic.bubble_case(nx, ny, nlay, 100e3, 100e3)
    d = Dycore(st)
    d.adj_enable()
    rng = np.random.default_rng(nx)
    for name, dtype in (('dp', torch.float64), ('vd', torch.float32)):
        t = torch.from_numpy(rng.normal(0, 1, (nlay, ny, nx))).to(dtype).cuda()
        a = t.cpu().numpy().astype(np.float64)
        d.upload_device(name, t)
        np.testing.assert_array_equal(d.get(name, halo=True), np.pad(a, ((0, 0), (H, H), (H, H)), mode='wrap'))
        out = torch.full_like(t, 7.0)
        d.download_device(name, out)
        assert torch.equal(out, t)
    t = torch.from_numpy(rng.normal(0, 1, (nlay, ny, nx))).cuda()
    d.adj_set_device('out', 'pt', t.data_ptr())
    np.testing.assert_array_equal(d.adj_get('out', 'pt'), np.pad(t.cpu().numpy(), ((0, 0), (H, H), (H, H))))
    out = torch.full_like(t, 7.0)
    d.adj_get_device('out', 'pt', out.data_ptr())
    d.sync()
    assert torch.equal(out, t)
    d.close()


@pytest.mark.parametrize('nx,ny,nlay', SIZES)
def test_finite_check(nx, ny, nlay):
    import torch
    st = ic.bubble_case(nx, ny, nlay, 100e3, 100e3)
    d = Dycore(st)
    good = torch.from_numpy(np.ascontiguousarray(st.pt)).cuda()
    d.upload_device('pt', good)
    assert d.check_stability()
    for x in sorted({0, nx // 2, nx - 1} | {q for q in (8, 64, 256, 384, 1024) if q < nx}):
        bad = good.clone()
        bad[nlay // 2, ny - 1, x] = np.inf
        d.upload_device('pt', bad)
        assert not d.check_stability(), x
    d.close()
