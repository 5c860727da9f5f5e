"""Shell sums, their adjoint and the overdensity at the edges of their loops:
odd and tiny row lengths, cross sums, lengths with remainders, NaN and misaligned
fields.

Bars: against float64 transforms 1e-5 of each shell's power (float32
transforms); the overdensity within one rounding of each of its two operations
(2^-22 of rho / mean + 1).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _conf(shape):
    import pmpp_b200 as pb
    return pb.Configuration(2.0, shape, 1, device="cuda")


def _shells(shape, ns):
    nx, ny, nz = shape
    md = lambda n: np.where(np.arange(n) < (n + 1) // 2, np.arange(n), np.arange(n) - n).astype(np.int64)
    n = np.meshgrid(md(nx), md(ny), np.arange(nz // 2 + 1), indexing="ij")
    return np.minimum(np.floor(np.sqrt(n[0]**2 + n[1]**2 + n[2]**2) + 1e-9).astype(int), ns - 1), n


def _reference(a, b, shape, ns, power):
    shell, (mx, my, mz) = _shells(shape, ns)
    nx, ny, nz = shape
    w = (np.sinc(mx / nx) * np.sinc(my / ny) * np.sinc(mz / nz))**-(2.0 * power)
    mult = np.where((mz == 0) | ((nz % 2 == 0) & (mz == nz // 2)), 1.0, 2.0)
    t = (a.real * b.real + a.imag * b.imag) * w * mult
    return np.bincount(shell.ravel(), t.ravel(), minlength=ns)[:ns]


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 3, 7), (9, 8, 65), (3, 2, 1), (2, 70, 130), (64, 64, 128),
                                   (64, 96, 128)])
@pytest.mark.parametrize("mas", [None, "CIC"])
def test_shell_sums_and_cross(shape, mas):
    from pmpp_b200 import power_spectrum as ps
    conf = _conf(shape)
    g = torch.Generator(device="cuda").manual_seed(3)
    x, y = (torch.randn(shape, generator=g, device="cuda") for _ in range(2))
    p = ps._mas(mas)
    got = [s.cpu().numpy() for s in ps._shell_sums(ps._spectrum(x, conf), conf, p, ps._spectrum(y, conf))]
    fa, fb = (np.fft.rfftn(t.cpu().numpy().astype(np.float64)) for t in (x, y))
    ns = ps.num_shells(conf)
    auto = [_reference(u, u, shape, ns, p) for u in (fa, fb)]
    bars = [1e-5 * v for v in (auto[0], auto[1], np.sqrt(auto[0] * auto[1]))]  # float32 transforms
    for i, ref in enumerate(auto + [_reference(fa, fb, shape, ns, p)]):
        assert np.all(np.abs(got[i] - ref) <= bars[i])


# rows whose window table along z is above 48 KB, and above all of shared memory
LONG = [(2, 3, 12288), (4, 1, 40001), (2, 1, 57344)]
# many rows on either side of the length from which a warp takes a row
EDGE = [(64, 33, 125), (64, 33, 126), (45, 45, 130), (48, 43, 130)]


@pytest.mark.parametrize("shape,cross,ns", [(LONG[0], True, 40), (LONG[1], False, 40), (LONG[2], False, 40),
                                            (LONG[2], True, 40), ((4, 2, 8192), True, 8533),
                                            ((2, 2, 40001), False, 25600), ((1030, 2, 12288), True, 40),
                                            ((2048, 1, 26000), False, 8000)] + [(e, True, 60) for e in EDGE])
@pytest.mark.parametrize("mas", [0, 2])
def test_shell_sums_of_long_rows(shape, cross, ns, mas):
    """Rows up to and beyond the length whose table fits beside the sums: FP64 products and sums of at most
    2^18 terms (bar 2^-34 of the sum of their magnitudes)."""
    from pmpp_b200 import power_spectrum as ps
    from pmpp_b200._lib import call
    from pmpp_b200.runtime import stream_handle
    g = torch.Generator(device="cuda").manual_seed(4)
    a, b = (torch.randn(shape[:2] + (shape[2] // 2 + 1, 2), generator=g, device="cuda") for _ in range(2))
    tab = ps._sinc_tables(_conf(shape), a.device)
    out = torch.empty((3, ns), dtype=torch.float64, device="cuda")
    ptr = lambda t: t.data_ptr() if cross else None
    call("pmb_pk_shells", a.data_ptr(), *shape, tab.data_ptr(), mas, ns, out[0].data_ptr(), ptr(b), ptr(out[1]),
         ptr(out[2]), stream_handle(a.device))
    t = np.split(tab.cpu().numpy().astype(np.float64), np.cumsum(shape[:2]))
    shell, (_, _, mz) = _shells(shape, ns)
    w = (t[0][:, None, None] * t[1][:, None] * t[2])**(-2.0 * mas)
    w = w * np.where((mz == 0) | ((shape[2] % 2 == 0) & (mz == shape[2] // 2)), 1.0, 2.0)
    ca, cb = (x.cpu().numpy().astype(np.float64) for x in (a, b))
    pairs = [(ca, ca)] + ([(cb, cb), (ca, cb)] if cross else [])
    for i, (x, y) in enumerate(pairs):
        v = (x[..., 0] * y[..., 0] + x[..., 1] * y[..., 1]) * w
        ref, mag = (np.bincount(shell.ravel(), z.ravel(), minlength=ns) for z in (v, np.abs(v)))
        assert np.all(np.abs(out[i].cpu().numpy() - ref) <= 2.0**-34 * mag)


@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 3, 7), (9, 8, 65), (3, 2, 1), (2, 70, 130), (2050, 1, 12288)] + LONG + EDGE)
def test_adjoint_rows(shape):
    """out = spec * 2 post W^-2p w[shell], in float64 and rounded once (bar 2^-22)."""
    from pmpp_b200 import power_spectrum as ps
    from pmpp_b200._lib import call
    from pmpp_b200.runtime import stream_handle
    conf = _conf(shape)
    ns = ps.num_shells(conf)
    rng = np.random.default_rng(7)
    nzh = shape[2] // 2 + 1
    spec = (rng.normal(size=shape[:2] + (nzh, )) + 1j * rng.normal(size=shape[:2] + (nzh, ))).astype(np.complex64)
    w = rng.normal(size=ns)
    x, wd = torch.from_numpy(spec).cuda(), torch.from_numpy(w).cuda()
    out = torch.full_like(x, float("nan"))
    tab = ps._sinc_tables(conf, x.device)
    call("pmb_pk_shells_adjoint", x.data_ptr(), *shape, tab.data_ptr(), 2, ns, wd.data_ptr(), 0.5, out.data_ptr(),
         stream_handle(x.device))
    t = np.split(tab.cpu().numpy().astype(np.float64), np.cumsum(shape[:2]))
    shell, _ = _shells(shape, ns)
    ref = spec.astype(complex) * (t[0][:, None, None] * t[1][:, None] * t[2])**-4.0 * w[shell]
    got = out.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 2.0**-22 * np.abs(ref))


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


@pytest.mark.parametrize("shape", [(8, 8, 8), (6, 10, 9)])
def test_loss_gradient_of_particles_on_cell_faces(shape):
    """The gradient of the P(k) loss against float64 autograd, with the mean density's own gradient, which
    reaches particles on a cell face only (their two-sided gradient takes one side's weights).  Bar: float32
    transforms and sums, 1e-5 of the largest component."""
    import pmpp_b200 as pb
    from pmpp_b200 import power_spectrum as ps
    conf = _conf(shape)
    rng = np.random.default_rng(5)
    n = conf.ptcl_num
    pmid = rng.integers(0, shape, size=(n, 3)).astype(np.int16)
    disp = (rng.integers(0, 2**12, size=(n, 3)) * 2.0**-11).astype(np.float32)  # exact in cells of 2
    disp[::3] = 0.0
    ns = ps.num_shells(conf)
    target = np.full(ns - 1, 50.0)
    loss, got = ps.pk_loss(pb.Particles(conf, torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda()), conf,
                           target)
    shell, (mx, my, mz) = _shells(shape, ns)
    w = (np.sinc(mx / shape[0]) * np.sinc(my / shape[1]) * np.sinc(mz / shape[2]))**-4.0
    w = w * np.where((mz == 0) | ((shape[2] % 2 == 0) & (mz == shape[2] // 2)), 1.0, 2.0)
    k, nmodes = ps.shell_statistics(conf)
    nmodes = torch.from_numpy(nmodes[:ns - 1].astype(np.float64))

    def reference(with_mean):
        d = torch.from_numpy(disp).double().requires_grad_(True)
        q = d / 2.0
        low = torch.floor(q).detach()
        f, base = q - low, torch.from_numpy(pmid).long() + low.long()
        rho = torch.zeros(int(np.prod(shape)), dtype=torch.float64)
        for b in range(8):
            bit = torch.tensor([b & 1, (b >> 1) & 1, b >> 2])
            i = torch.remainder(base + bit, torch.tensor(shape))
            rho = rho.index_add(0, (i[:, 0] * shape[1] + i[:, 1]) * shape[2] + i[:, 2],
                                (1 - (f - bit).abs()).prod(-1))
        mean = rho.mean() if with_mean else rho.mean().detach()
        spec = torch.fft.rfftn((rho / mean - 1).reshape(shape))
        p = (spec.real**2 + spec.imag**2) * torch.from_numpy(w)
        s = torch.zeros(ns, dtype=torch.float64).index_add(0, torch.from_numpy(shell).reshape(-1), p.reshape(-1))[1:]
        pk = s / nmodes * (8.0 / np.prod(shape))
        lr = torch.log(pk[nmodes > 0] / 50.0)
        out = (lr**2).mean()
        return float(out), torch.autograd.grad(out, d)[0].numpy()

    ref_loss, ref = reference(True)
    bar = 1e-5 * np.abs(ref).max()
    np.testing.assert_allclose(loss, ref_loss, rtol=1e-5)
    assert np.abs(got.cpu().numpy() - ref).max() <= bar
    assert np.abs(reference(False)[1] - ref).max() > 100 * bar  # the mean's share is seen
