"""Shell sums, their adjoint and the overdensity at the edges of their loops:
odd and tiny row lengths, meshes of the FFT pass chain (blocked rows) against
rows in order, cross sums, lengths with remainders, NaN and misaligned fields.

Bars: against float64 transforms 1e-5 of each shell's power (float32
transforms); between the layouts the same float64 terms in another order, 1e-12;
the adjoint is element by element, so exact; the overdensity within one rounding
of each of its two operations (2^-22 of rho / mean + 1)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _conf(shape):
    import pmpp_b200 as pb
    return pb.Configuration(2.0, shape, 1, device="cuda")


def _reference(a, b, shape, ns, power):
    nx, ny, nz = shape
    md = lambda n: np.where(np.arange(n) < (n + 1) // 2, np.arange(n), np.arange(n) - n).astype(np.int64)
    mx, my, mz = np.meshgrid(md(nx), md(ny), np.arange(nz // 2 + 1), indexing="ij")
    shell = np.minimum(np.floor(np.sqrt(mx * mx + my * my + mz * mz) + 1e-9).astype(int), ns - 1)
    w = (np.sinc(mx / nx) * np.sinc(my / ny) * np.sinc(mz / nz))**-(2.0 * power)
    mult = np.where((mz == 0) | ((nz % 2 == 0) & (mz == nz // 2)), 1.0, 2.0)
    t = (a.real * b.real + a.imag * b.imag) * w * mult
    add = lambda v: np.bincount(shell.ravel(), v.ravel(), minlength=ns)[:ns]
    return add(t)


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 3, 7), (9, 8, 65), (3, 2, 1), (2, 70, 130), (64, 64, 128),
                                   (64, 96, 128)])
@pytest.mark.parametrize("mas", [None, "CIC"])
def test_shell_sums_both_layouts_and_cross(shape, mas):
    from pmpp_b200 import _lib, power_spectrum as ps
    conf = _conf(shape)
    g = torch.Generator(device="cuda").manual_seed(3)
    x, y = (torch.randn(shape, generator=g, device="cuda") for _ in range(2))
    p = ps._mas(mas)
    res = {}
    try:
        for on in (True, False):
            _lib.set_pmfft(on)
            res[on] = [s.cpu().numpy() for s in ps._shell_sums(ps._spectrum(x, conf), conf, p, ps._spectrum(y, conf))]
    finally:
        _lib.set_pmfft(True)
    fa, fb = (np.fft.rfftn(t.cpu().numpy().astype(np.float64)) for t in (x, y))
    ns = ps.num_shells(conf)
    auto = [_reference(u, u, shape, ns, p) for u in (fa, fb)]
    bars = [1e-5 * v for v in (auto[0], auto[1], np.sqrt(auto[0] * auto[1]))]  # float32 transforms
    for i, ref in enumerate(auto + [_reference(fa, fb, shape, ns, p)]):
        for on in (True, False):
            assert np.all(np.abs(res[on][i] - ref) <= bars[i])


@pytest.mark.parametrize("shape", [(64, 64, 128), (96, 64, 128)])
def test_blocked_layout_equals_rows_in_order(shape):
    from pmpp_b200 import power_spectrum as ps
    from pmpp_b200._lib import call
    from pmpp_b200.runtime import stream_handle
    nx, ny, nz = shape
    nzh = nz // 2 + 1
    conf = _conf(shape)
    x = torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda")
    spec, blocked = ps._spectrum(x, conf)
    assert blocked
    rows = lambda t: t.view(ny // 32, nx, 32, -1).permute(1, 0, 2, 3).reshape(nx, ny, -1)
    flat = rows(spec)[..., :nzh].contiguous()
    a, _, _ = ps._shell_sums((spec, 1), conf, 2)
    b, _, _ = ps._shell_sums((flat, 0), conf, 2)
    np.testing.assert_allclose(a.cpu().numpy(), b.cpu().numpy(), rtol=1e-12)
    ns = ps.num_shells(conf)
    w = torch.randn(ns, dtype=torch.float64, device="cuda")
    tab = ps._sinc_tables(conf, x.device)
    s = stream_handle(x.device)
    out = [torch.full_like(t, float("nan")) for t in (spec, flat)]
    for t, o, blk in ((spec, out[0], 1), (flat, out[1], 0)):
        call("pmb_pk_shells_adjoint2", t.data_ptr(), nx, ny, nz, blk, tab.data_ptr(), 2, ns, w.data_ptr(), 0.5,
             o.data_ptr(), s)
    got = rows(out[0])
    assert torch.equal(got[..., :nzh], out[1]) and not bool(got[..., nzh:].abs().sum())
    call("pmb_pk_shells_adjoint2", spec.data_ptr(), nx, ny, nz, 1, tab.data_ptr(), 2, ns, w.data_ptr(), 0.5,
         spec.data_ptr(), s)  # in place
    assert torch.equal(rows(spec), got)


def test_misaligned_field_stays_refused():
    from pmpp_b200 import power_spectrum as ps
    from pmpp_b200._lib import PMBError
    conf = _conf((64, 64, 128))
    buf = torch.zeros(64 * 64 * 128 + 1, device="cuda")
    with pytest.raises(PMBError):
        ps.delta_to_pk(buf[1:].view(64, 64, 128), conf)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4097, 100003])
@pytest.mark.parametrize("at", [0, 1])
def test_overdensity_remainders(n, at):
    from pmpp_b200._lib import call
    from pmpp_b200.runtime import stream_handle
    rho = torch.rand(n + 1, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda")[at:at + n] + 0.5
    buf = torch.zeros(n + 5, device="cuda")
    src = buf[at:at + n].copy_(rho)
    out = torch.full((n + 5, ), 7.0, device="cuda")
    tot = src.double().sum().reshape(1)
    call("pmb_overdensity", src.data_ptr(), out[at:].data_ptr(), n, tot.data_ptr(), stream_handle(rho.device))
    r = rho.cpu().numpy().astype(np.float64)
    r /= r.mean()
    assert np.all(np.abs(out[at:at + n].cpu().numpy() - (r - 1)) <= 2.0**-22 * (r + 1))
    assert bool((out[:at] == 7).all()) and bool((out[at + n:] == 7).all())
    if n > 2:
        src[n - 1] = float("nan")
        call("pmb_overdensity", src.data_ptr(), out[at:].data_ptr(), n, tot.data_ptr(), stream_handle(rho.device))
        assert bool(out[at + n - 1].isnan()) and not bool(out[at:at + n - 1].isnan().any())
