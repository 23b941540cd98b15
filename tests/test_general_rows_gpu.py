"""GPU tests of the general transform's row passes and of the layout of its
spectra: half spectra of 8 to 16 bins (FFT3D pads their rows to whole 64
bytes, the plain method packs them, so that rows start on 16-byte boundaries
or not), rows that do not fill a tile, padding boxes that cut rows, are empty
or not there, stored spectra of the packed layout.  Tolerance: the general
methods' parity bound against the FP64 oracle (relative L2 1e-5)."""
import numpy as np
import pytest

import oracle
import vfd

pytestmark = pytest.mark.gpu

REL_L2 = 1e-5
NONE = (np.zeros(0, np.int32), np.zeros(0, np.float32))


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    return float(np.sqrt(((a - b) ** 2).sum() / max((b ** 2).sum(), 1e-300)))


@pytest.mark.parametrize("fx", [14, 16, 18, 20, 24, 28, 30])
@pytest.mark.parametrize("method", [vfd.METHOD_FFT3D, vfd.METHOD_PLAIN])
def test_half_spectrum_lengths(gpu, fx, method):
    nx, ny, nz, r = fx - 3, 11, 7, 3
    for pad, epi in ((vfd.PAD_ZERO, 0), (vfd.PAD_CONSTANT_VF, nx - 2), (vfd.PAD_CONSTANT_VF, nx), (vfd.PAD_CONSTANT_VF, 1)):
        u = vfd.synth_field(5, 0, 0, (nz, ny, nx))
        b = 2e-4 if pad == vfd.PAD_CONSTANT_VF else 0.0
        with vfd.World(nx, ny, nz, [vfd.field_params(0.8, 0.03, radius=r, baseline=b)], pad_mode=pad, epi_boundary=epi,
                       fft=(fx, 15, 12), method=method) as w:
            w.upload(0, u)
            w.tick(1)
            out, mass = w.download(0), w.mass()[0]
        ref = oracle.tick(u, 0.8, 0.03, 1, *NONE, b=float(np.float32(b)), pad_mode=pad, epi=epi, radius3=r)
        assert rel_l2(out, ref) <= REL_L2, (fx, pad, epi)
        s = out.astype(np.float64).sum()
        assert abs(mass["total"] - s) <= 1e-6 * max(abs(s), 1e-30)


@pytest.mark.parametrize("fx", [14, 16, 18, 28])
def test_stored_spectra(gpu, fx):
    """A window's spectrum, read back packed and stored again, gives the
    window's own results; its window comes back from it."""
    fft, (nx, ny, nz) = (fx, 15, 12), (fx - 3, 11, 7)
    rng = np.random.default_rng(fx)
    win = rng.random((5, 3, 7)).astype(np.float32)
    win /= win.sum()
    u = vfd.synth_field(6, 0, 0, (nz, ny, nx))
    outs = []
    spec = vfd.window_spectrum(win, fft)
    want = np.zeros((12, 15, fx))
    for z in range(5):
        for y in range(3):
            for x in range(7):
                want[(z - 2) % 12, (y - 1) % 15, (x - 3) % fx] += win[z, y, x]
    assert rel_l2(spec.view(np.float32), np.fft.rfftn(want).view(np.float64)) <= REL_L2
    assert rel_l2(vfd.spectrum_window(spec, fx, win.shape), win) <= REL_L2
    for stored in (False, True):
        with vfd.World(nx, ny, nz, [vfd.field_params(1.0, 0.0, radius=3)] * 2, fft=fft, method=vfd.METHOD_FFT3D) as w:
            for f in range(2):
                w.upload(f, u)
                w.set_spectrum(f, spec) if stored else w.set_window(f, win)
            w.tick(1)
            outs.append([w.download(f) for f in range(2)])
    for a, b in zip(outs[0] + outs[0], outs[1] + outs[1][::-1]):
        np.testing.assert_array_equal(a, b)
