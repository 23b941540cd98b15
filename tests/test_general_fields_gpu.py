"""GPU tests of the general transform's launches of several fields and of its
update epilogue: FFT lengths whose last inverse factor is 2, 3, odd, even and
24, the 16-line kernels and the Stockham kernels, fields with and without a
dChem array in one tick, more fields than a launch holds.  Tolerance: the
general methods' parity bound against the FP64 oracle (relative L2 1e-5)."""
import numpy as np
import pytest

import oracle
import vfd

pytestmark = pytest.mark.gpu

REL_L2 = 1e-5


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    return float(np.sqrt(((a - b) ** 2).sum() / max((b ** 2).sum(), 1e-300)))


def check(grid, fft, nf, substeps=1, with_d=None, pad=vfd.PAD_CONSTANT_VF):
    import torch
    nx, ny, nz = grid
    epi = nx - 2
    sig = [0.6 + 0.07 * f for f in range(nf)]
    params = [vfd.field_params(sig[f], 0.02, radius=4, baseline=1e-4 * (f + 1)) for f in range(nf)]
    decay = [0.9 + 0.01 * f for f in range(nf)]
    with vfd.World(nx, ny, nz, params, pad_mode=pad, epi_boundary=epi, fft=fft, method=vfd.METHOD_FFT3D) as w:
        us = [vfd.synth_field(11, 0, f, (nz, ny, nx)) for f in range(nf)]
        ds = [torch.rand((nz, ny, nx), device="cuda") * 1e-3 if with_d is None or f in with_d else None for f in range(nf)]
        d0 = [None if d is None else d.cpu().numpy() for d in ds]
        for f, u in enumerate(us):
            w.upload(f, u)
        w.tick_update(decay, [0 if d is None else d.data_ptr() for d in ds], substeps)
        outs = [w.download(f) for f in range(nf)]
        mass = w.mass()
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    for f in range(nf):
        t = oracle.tick(us[f], sig[f], 0.02, substeps, *none, b=float(np.float32(1e-4 * (f + 1))), pad_mode=pad, epi=epi,
                        radius3=4)
        ref = t * float(np.float32(decay[f])) + (0 if d0[f] is None else d0[f])
        assert rel_l2(outs[f], ref) <= REL_L2, (fft, f)
        s = outs[f].astype(np.float64).sum()
        assert abs(mass[f]["total"] - s) <= 1e-6 * abs(s)
        if ds[f] is not None:
            assert float(ds[f].abs().max()) == 0.0


# x lengths 42 = 6 x 7, 60 = 6 x 10, 28 = 4 x 7, 18 = 3 x 6, 48 = 6 x 8, 576 = 24 x 24; 50 = 5 x 10
@pytest.mark.parametrize("grid,fft", [((37, 20, 15), (42, 27, 20)), ((55, 13, 20), (60, 18, 24)), ((24, 30, 9), (28, 35, 18)),
                                      ((14, 14, 14), (18, 18, 18)), ((43, 40, 21), (48, 50, 28)),
                                      ((571, 9, 7), (576, 15, 14))])
@pytest.mark.parametrize("nf", [1, 3])
def test_update_epilogue_lengths(gpu, grid, fft, nf):
    check(grid, fft, nf)


def test_sixteen_line_and_stockham_kernels(gpu):
    check((700, 6, 8), (720, 14, 14), 3)      # 720 = 24 x 30: 16-line rows
    check((680, 6, 8), (686, 14, 14), 3)      # 2 * 7^3: no split, Stockham rows
    check((20, 6, 660), (28, 14, 672), 2)     # long z lines


def test_fields_with_and_without_dchem(gpu):
    check((40, 21, 18), (48, 28, 24), 7, substeps=2, with_d=(1, 2, 6))


def test_more_fields_than_a_launch_holds(gpu):
    check((33, 20, 17), (40, 24, 21), 11)


@pytest.mark.parametrize("method,kind", [(vfd.METHOD_FFT3D, k) for k in ("same", "overlapping", "own", "next", "previous")]
                         + [(vfd.METHOD_SEPARABLE, "same"), (vfd.METHOD_SEPARABLE, "overlapping")])
def test_shared_dchem(gpu, method, kind):
    """Device dChem arrays that fields share, or that are fields of the world:
    the fields are updated in order, so the first takes the values and the
    others find zeros.  The grid's spectra fit one launch of several fields."""
    import torch
    nx, ny, nz, nf = 40, 30, 22, 4
    V = nx * ny * nz
    sig = [0.6 + 0.07 * f for f in range(nf)]
    decay = [np.float32(0.9 + 0.01 * f) for f in range(nf)]
    us = [vfd.synth_field(3, 0, f, (nz, ny, nx)) for f in range(nf)]
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    buf = torch.rand((2 * V,), device="cuda") * 1e-3
    # one run of memory: the world's fields, then the two arrays
    mem = np.concatenate([u.ravel() for u in us] + [buf.cpu().numpy()]).astype(np.float64)
    D = nf * V
    at = {"same": [D, D, D + V, D], "overlapping": [D, D + V // 3, D + V, None], "own": [0, V, 2 * V, D],
          "next": [V, 2 * V, D, None], "previous": [D, 0, V, 2 * V]}[kind]
    with vfd.World(nx, ny, nz, [vfd.field_params(s, 0.02, radius=4) for s in sig], method=method) as w:
        for f, u in enumerate(us):
            w.upload(f, u)
        ptr = [None if a is None else w.device_ptr(0) + 4 * a if a < D else buf.data_ptr() + 4 * (a - D) for a in at]
        w.tick_update(decay, [p or 0 for p in ptr], 1)
        outs = np.concatenate([w.download(f).ravel() for f in range(nf)] + [buf.cpu().numpy()])

    def tick(f):
        u = mem[f * V:(f + 1) * V].astype(np.float32).reshape(nz, ny, nx)
        return oracle.tick(u, sig[f], 0.02, 1, *none, radius3=4).ravel() * float(decay[f])

    def update(f, t):
        d = np.zeros(V) if at[f] is None else mem[at[f]:at[f] + V].copy()
        if at[f] is not None:
            mem[at[f]:at[f] + V] = 0.0
        mem[f * V:(f + 1) * V] = d + t

    for f in range(nf):
        update(f, tick(f))
    assert rel_l2(outs, mem) <= REL_L2
    for f in range(nf):
        assert rel_l2(outs[f * V:(f + 1) * V], mem[f * V:(f + 1) * V]) <= REL_L2, f
    np.testing.assert_array_equal(outs[D:] == 0, mem[D:] == 0)


@pytest.mark.parametrize("method", [vfd.METHOD_FFT3D, vfd.METHOD_SEPARABLE])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "shared", "partial"])
def test_update_host_buffers(gpu, method, kind):
    """vfd_diffuse_update_host zeroes dChem in pinned buffers by copies from the
    device, in others on the host; a buffer that several fields share is read
    by all of them before it is zeroed."""
    import torch
    nx, ny, nz, nf = 40, 30, 22, 4
    sig = [0.7 + 0.2 * f for f in range(nf)]
    decay = [0.9] * nf
    rng = np.random.default_rng(3)

    def buffers(n):
        a = [rng.random((nz, ny, nx), dtype=np.float32) * np.float32(1e-3) for _ in range(n)]
        return a if kind == "pageable" else [torch.from_numpy(x).pin_memory().numpy() for x in a]

    p, d = buffers(nf), buffers(nf)
    if kind == "shared":
        d = [d[0]] * nf
    p0, d0 = [x.copy() for x in p], [x.copy() for x in d]
    params = [vfd.field_params(s, 0.02) for s in sig]
    with vfd.World(nx, ny, nz, params, method=method) as w:
        if kind == "partial":
            import ctypes as C
            ps = (C.c_void_p * nf)(*[x.ctypes.data for x in p])
            ds = (C.c_void_p * nf)(*[x.ctypes.data if f % 2 else None for f, x in enumerate(d)])
            dec = np.array(decay, np.float32)
            assert vfd.lib().vfd_diffuse_update_host(w.handle, ps, ds, dec.ctypes.data, 1) == 0
        else:
            w.diffuse_update_host(p, d, decay)
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    for f in range(nf):
        has = kind != "partial" or f % 2
        ref = oracle.tick(p0[f], sig[f], 0.02, 1, *none) * float(np.float32(0.9)) + (d0[f] if has else 0)
        assert rel_l2(p[f], ref) <= REL_L2, f
        if has:
            assert not d[f].any()
        else:
            np.testing.assert_array_equal(d[f], d0[f])
