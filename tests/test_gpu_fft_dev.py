"""Device-resident transforms (db_fft_xz_to_fourier_dev / _physical_dev) on
device arrays in the reference layout, against the host-array forms on the
same fields: bit-identical on FP64 and mixed-precision contexts, the padding
of the physical layout left as it was in both."""
import numpy as np
import pytest

from _util import config0_params, grid_for

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("prec", [0, 1])
def test_device_transforms_match_host_forms(prec):
    from diablo3_b200.channel import Channel
    p = config0_params(nx=32, ny=33, nz=32, precision=prec)
    ch = Channel(p, grid_for(p))
    rng = np.random.default_rng(7)
    phys = rng.standard_normal(ch.new_real().shape)   # padding holds values too
    # forward
    spec_host = ch.fft_xz_to_fourier(phys.copy()).copy()
    d = torch.from_numpy(phys.copy()).cuda()
    torch.cuda.synchronize()
    ch.fft_xz_to_fourier_dev(d)
    torch.cuda.synchronize()
    spec_dev = d.cpu().numpy().reshape(-1).view(np.complex128).reshape(spec_host.shape)
    assert np.array_equal(spec_dev, spec_host)
    # inverse, from a spectral array whose unretained entries hold values
    # (both forms ignore them)
    spec = spec_host.copy()
    nkx, nkzp = p.nx // 3, 2 * (p.nz // 3) + 1
    spec[:, :, nkx + 1:] = rng.standard_normal(spec[:, :, nkx + 1:].shape)
    spec[:, nkzp:, :] = rng.standard_normal(spec[:, nkzp:, :].shape)
    phys_host = ch.fft_xz_to_physical(spec.copy()).copy()
    d2 = torch.from_numpy(spec.copy()).cuda()
    torch.cuda.synchronize()
    ch.fft_xz_to_physical_dev(d2)
    torch.cuda.synchronize()
    phys_dev = d2.cpu().numpy().reshape(-1).view(np.float64).reshape(phys_host.shape)
    assert np.array_equal(phys_dev, phys_host)
    # the forward transform of the band-limited result gives the same modes
    d3 = torch.from_numpy(phys_dev.copy()).cuda()
    torch.cuda.synchronize()
    ch.fft_xz_to_fourier_dev(d3)
    torch.cuda.synchronize()
    again = d3.cpu().numpy().reshape(-1).view(np.complex128).reshape(spec_host.shape)
    tol = 1e-12 if prec == 0 else 1e-5
    assert np.abs(again - spec_host).max() <= tol * np.abs(spec_host).max()
    ch.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [
    (16, 9, 32), (16, 9, 512),      # sequences of two threads; one and several blocks of rows a plane
    (64, 33, 256), (512, 17, 512),  # several items a CTA (1216 of them at 512, up to 5 each): both buffers, both parities
    (512, 11, 16), (1024, 5, 32),   # sequences over more than a warp, one item a CTA
])
def test_device_transforms_over_sizes(n, prec):
    """Bit-identical to the host forms, which stage compact rows."""
    from diablo3_b200.channel import Channel
    p = config0_params(nx=n[0], ny=n[1], nz=n[2], precision=prec)
    with Channel(p, grid_for(p)) as ch:
        phys = np.random.default_rng(3).standard_normal(ch.new_real().shape)
        d = torch.from_numpy(phys.copy()).cuda()
        torch.cuda.synchronize()
        ch.fft_xz_to_fourier_dev(d)
        torch.cuda.synchronize()
        spec = ch.fft_xz_to_fourier(phys).copy()
        assert np.array_equal(d.cpu().numpy().reshape(-1).view(np.complex128).reshape(spec.shape), spec)
        ch.fft_xz_to_physical_dev(d)
        torch.cuda.synchronize()
        back = ch.fft_xz_to_physical(spec)
        assert np.array_equal(d.cpu().numpy()[:, :p.nz, :p.nx], back[:, :p.nz, :p.nx])


@pytest.mark.parametrize("prec", [0, 1])
def test_misaligned_device_array_is_refused(prec):
    """A float64 view 8 bytes off: an error code from both calls, nothing launched."""
    from diablo3_b200.channel import Channel
    from diablo3_b200.lib import DiabloError
    p = config0_params(nx=16, ny=9, nz=16, precision=prec)
    with Channel(p, grid_for(p)) as ch:
        d = torch.ones(ch.new_real().size + 1, dtype=torch.float64, device="cuda")
        for call in (ch.fft_xz_to_fourier_dev, ch.fft_xz_to_physical_dev):
            with pytest.raises(DiabloError, match="aligned"):
                call(d[1:])
        torch.cuda.synchronize()
        assert bool((d == 1.0).all())


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [(128, 63, 64), (256, 33, 64), (64, 34, 32), (128, 33, 256)])
def test_repeated_transforms_give_the_same_bits(n, prec):
    """A CTA of the z-passes transforms two planes in turn: nothing of one may reach the other's stores (1 in 15 to 1
    in 500 of the FP32 forward transforms of the first two sizes had a wrong row once)."""
    from diablo3_b200.channel import Channel
    p = config0_params(nx=n[0], ny=n[1], nz=n[2], precision=prec)
    with Channel(p, grid_for(p)) as ch:
        phys = torch.from_numpy(np.random.default_rng(5).standard_normal(ch.new_real().shape)).cuda()
        spec = torch.from_numpy(ch.fft_xz_to_fourier(phys.cpu().numpy()).view(np.float64).reshape(phys.shape).copy()).cuda()
        d, first, bad = phys.clone(), None, 0
        for _ in range(1500):
            out = []
            for src, call in ((phys, ch.fft_xz_to_fourier_dev), (spec, ch.fft_xz_to_physical_dev)):
                d.copy_(src)
                torch.cuda.synchronize()
                call(d)
                torch.cuda.synchronize()
                out.append(d.view(torch.int64).clone())
            if first is None:
                first = out
            bad += sum(not torch.equal(a, b) for a, b in zip(out, first))
        assert bad == 0
