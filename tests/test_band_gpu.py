"""GPU tests of the banded-product passes (m substeps folded into one operator
per axis, applied on the tensor cores) at the sizes where their tiling,
operators and folding change: lines of one block, one more and one less,
partly filled tiles, the three ways input blocks are copied, narrow and wide
kernels, several groups of folded substeps, the padding rule's affine part.

Tolerance: a pass rounds its inputs (relative to the line's offset), three
parts of value and weight (2^-24 each), a K / 16-step accumulation whose
truncation is relative to values about the offset, and the sum with the
offset's product: at most 4 units of 2^-24 of the field's level; three passes
a group and the final decay and deposit give 14 * 2^-24 = 8.4e-7 a group."""
import numpy as np
import pytest

import oracle
import vfd

pytestmark = pytest.mark.gpu

PER_GROUP = 14 * 2.0 ** -24


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    return float(np.sqrt(((a - b) ** 2).sum() / max((b ** 2).sum(), 1e-300)))


def check(grid, sig, substeps, groups=1, pad=vfd.PAD_ZERO, epi=0, base=0.0, dec=0.04, radius=None, nf=2, seed=9):
    nx, ny, nz = grid
    V = nx * ny * nz
    params = [vfd.field_params(sig, dec, radius=radius, baseline=base * (f + 1)) for f in range(nf)]
    ins = []
    with vfd.World(nx, ny, nz, params, pad_mode=pad, epi_boundary=epi) as w:
        for f in range(nf):
            u = vfd.synth_field(seed, 1, f, (nz, ny, nx))
            idx, amt = vfd.synth_sources(seed, 1, f, 23, V)
            ins.append((u, idx, amt))
            w.upload(f, u)
            w.set_sources(f, idx, amt)
        w.tick(substeps)
        outs = [w.download(f) for f in range(nf)]
        mass = w.mass()
    for f, (u, idx, amt) in enumerate(ins):
        b = float(np.float32(base * (f + 1)))
        ref = oracle.tick(u, sig, dec, substeps, idx, amt, b=b, pad_mode=pad, epi=epi, radius3=radius)
        e = rel_l2(outs[f], ref)
        assert e <= groups * PER_GROUP, (grid, sig, substeps, f, e)
        m, s = mass[f], outs[f].astype(np.float64).sum()
        scale = max(abs(m["input_sum"]), abs(s), 1e-30)
        assert abs(m["input_sum"] - m["conv_sum"] - sum(m["leaked"])) <= 1e-6 * scale
        assert abs(m["total"] - s) <= 1e-6 * max(abs(s), 1e-30)


# x lines of one block, its neighbours and several; nx % 4 != 0 (4-byte
# copies), % 4 == 0 (16-byte copies along y), % 32 == 0 (bulk tensor copies)
@pytest.mark.parametrize("grid", [(64, 5, 3), (63, 9, 4), (65, 3, 7), (68, 70, 9), (128, 66, 3), (96, 64, 65),
                                  (129, 33, 1), (1, 64, 130), (260, 4, 11)])
@pytest.mark.parametrize("substeps", [1, 10])
def test_line_lengths_and_copies(gpu, grid, substeps):
    check(grid, 1.3, substeps)


# half-widths of 4 and 8 up to the widest operator (radius 56), and kernels
# wider than short lines
@pytest.mark.parametrize("radius", [1, 4, 9, 17, 33, 56])
def test_kernel_widths(gpu, radius):
    check((200, 36, 40), radius / 3.0, 1, radius=radius)


# groups (at most): sigma 2.6 folds 14 substeps (half-width <= 56), 0.6 folds 16
@pytest.mark.parametrize("sigma,substeps,groups", [(2.6, 11, 1), (2.6, 12, 2), (2.6, 14, 1), (2.6, 15, 2), (2.6, 25, 3), (0.6, 16, 1), (0.6, 17, 2),
                                                   (5.0, 3, 1), (5.0, 7, 3)])
def test_folded_groups(gpu, sigma, substeps, groups):
    check((140, 70, 68), sigma, substeps, groups=groups)


@pytest.mark.parametrize("substeps", [1, 2, 10, 19])
@pytest.mark.parametrize("epi", [1, 2, 65, 130, 200])
def test_padding_rule(gpu, substeps, epi):
    check((132, 20, 35), 1.1, substeps, groups=(substeps + 15) // 16, pad=vfd.PAD_CONSTANT_VF, epi=epi, base=3e-4)


def test_signs_and_scales(gpu):
    """Fields of either sign and of scales 1e-20 and 1e20 (the offset and the
    bf16 parts keep FP32's range), one field each in one launch."""
    nx, ny, nz = 72, 40, 33
    rng = np.random.default_rng(4)
    us = [(rng.standard_normal((nz, ny, nx)) * s).astype(np.float32) for s in (1.0, 1e-20, 1e20)]
    with vfd.World(nx, ny, nz, [vfd.field_params(1.4, 0.02)] * 3) as w:
        for f, u in enumerate(us):
            w.upload(f, u)
        w.tick(4)
        outs = [w.download(f) for f in range(3)]
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    for u, o in zip(us, outs):
        ref = oracle.tick(u, 1.4, 0.02, 4, *none)
        # four substeps shrink unit noise to about 1/30: the bound is on the input's scale
        err = np.sqrt(((o - ref) ** 2).sum() / (u.astype(np.float64) ** 2).sum())
        assert err <= PER_GROUP


def test_non_finite_values_stay_local(gpu):
    """A NaN reaches its own lines only; the rest of the field is untouched."""
    nx, ny, nz = 160, 24, 70
    u = vfd.synth_field(2, 0, 0, (nz, ny, nx))
    bad = u.copy()
    bad[40, 12, 20] = np.nan
    outs = []
    for v in (u, bad):
        with vfd.World(nx, ny, nz, [vfd.field_params(0.6, 0.0)]) as w:
            w.upload(0, v)
            w.tick(1)
            outs.append(w.download(0))
    hit = ~np.isfinite(outs[1])
    assert hit[40, 12, 20]
    # x lines of the window's blocks, every y of the line block, z blocks likewise: never the far x half
    assert not hit[:, :, 136:].any()
    np.testing.assert_array_equal(outs[0][~hit], outs[1][~hit])


def test_single_field_and_world_launches_agree(gpu):
    """vfd_diffuse_host runs one field a launch, a batch all worlds in one."""
    grid, sig = (100, 41, 37), [0.9, 1.7, 2.3]
    nx, ny, nz = grid
    params = [vfd.field_params(s, 0.03) for s in sig]
    us = [vfd.synth_field(6, 0, f, (nz, ny, nx)) for f in range(3)]
    with vfd.World(nx, ny, nz, params) as w, vfd.World(nx, ny, nz, params) as v, vfd.World(40, 30, 20, params) as o:
        for f, u in enumerate(us):
            w.upload(f, u)
            v.upload(f, u)
            o.upload(f, vfd.synth_field(7, 0, f, (20, 30, 40)))
        w.tick(5)
        outs = [w.download(f) for f in range(3)]
        with vfd.Batch([o, v]) as b:
            b.tick(5)
        for f in range(3):
            np.testing.assert_array_equal(outs[f], v.download(f))
        host = [np.empty_like(u) for u in us]
        w.diffuse_host(us, host, 5)
    for f in range(3):
        np.testing.assert_array_equal(outs[f], host[f])


def test_batch_results_do_not_depend_on_neighbours(gpu):
    """Worlds on banded products, on FFT passes (a single substep of a large
    world with narrow kernels; pinned passes) and with several groups of
    folded substeps share a batch: each result equals its own single tick."""
    vfd.autotune_clear()
    try:
        vfd.autotune_set(44, 40, 36, [vfd.field_params(1.0, 0.02)] * 2, [{"method": "overlap_save"}] * 3)
        specs = [((44, 40, 36), 1.0), ((176, 160, 96), 0.9), ((90, 33, 70), 2.6), ((64, 64, 32), 0.7)]
        for substeps in (1, 12):
            worlds, singles = [], []
            for i, (g, sig) in enumerate(specs):
                for out in (worlds, singles):
                    w = vfd.World(*g, [vfd.field_params(sig, 0.02)] * 2)
                    for f in range(2):
                        w.upload(f, vfd.synth_field(3, i, f, g[::-1]))
                    out.append(w)
            with vfd.Batch(worlds) as b:
                for _ in range(3):  # directly, captured, replayed
                    b.tick(substeps)
                b.tick(3)
                b.tick(substeps)
            for w, v in zip(worlds, singles):
                for n in (substeps,) * 3 + (3, substeps):
                    v.tick(n)
                for f in range(2):
                    np.testing.assert_array_equal(w.download(f), v.download(f))
                got, ref = w.mass(), v.mass()
                for f in range(2):
                    assert got[f]["total"] == pytest.approx(ref[f]["total"], rel=1e-12)
                    assert got[f]["input_sum"] == pytest.approx(ref[f]["input_sum"], rel=1e-12)
                w.close()
                v.close()
    finally:
        vfd.autotune_clear()


# Fields of a wide range.  What an output may be off by is relative to the
# values its blocks hold: the sum of |weight x value| and the mean of a block of
# 64 that holds it (the offset), 14 * 2^-24 of each a group.  A window of blocks
# reaches at most 192 positions from an output.
REACH = 192
LONG = 520
GRIDS = [(LONG, 6, 5), (7, LONG, 4), (5, 6, LONG)]


def along(axis, n):
    """Positions along `axis` as a (nz, ny, nx) array that broadcasts."""
    return np.arange(n).reshape([-1 if a == 2 - axis else 1 for a in range(3)])


def run_once(grid, u, sig, substeps, dec=0.0):
    with vfd.World(*grid, [vfd.field_params(sig, dec)]) as w:
        w.upload(0, u)
        w.tick(substeps)
        out, mass = w.download(0), w.mass()[0]
    ref = oracle.tick(u, sig, dec, substeps, np.zeros(0, np.int32), np.zeros(0, np.float32))
    return out.astype(np.float64), ref, mass


# half-widths of 8 (one substep of sigma 2.6), 32 and 48 (ten of 1.3 and of 2.6)
WIDE = [(2.6, 1), (1.3, 10), (2.6, 10)]


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sigma,substeps", WIDE)
def test_single_voxel_in_the_middle(gpu, axis, sigma, substeps):
    """One voxel of 1 at the middle of every axis, nothing else: the result is
    as accurate as a dense field's, and zero where no block sees the voxel."""
    grid = GRIDS[axis]
    u = np.zeros(grid[::-1], np.float32)
    u[grid[2] // 2, grid[1] // 2, grid[0] // 2] = 1.0
    out, ref, mass = run_once(grid, u, sigma, substeps)
    assert rel_l2(out, ref) <= 2 * PER_GROUP  # its own products' and the offset's
    assert abs(out.sum() - ref.sum()) <= 1e-6 * ref.sum()
    far = np.broadcast_to(np.abs(along(axis, LONG) - LONG // 2) > REACH, out.shape)
    assert far.any() and not out[far].any()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sigma,substeps", WIDE)
@pytest.mark.parametrize("at", [0, LONG // 2 - 30, LONG - 60])
def test_plume_leaves_zeros_alone(gpu, axis, sigma, substeps, at):
    """60 voxels of about 0.5 at either end or in the middle, zeros elsewhere."""
    grid = GRIDS[axis]
    p = along(axis, LONG)
    u = np.where((p >= at) & (p < at + 60), 0.5 + vfd.synth_field(4, 0, 0, grid[::-1]), 0.0).astype(np.float32)
    out, ref, mass = run_once(grid, u, sigma, substeps)
    assert rel_l2(out, ref) <= PER_GROUP
    assert abs(out.sum() - ref.sum()) <= 1e-6 * ref.sum()
    far = np.broadcast_to((p < at - REACH) | (p >= at + 60 + REACH), out.shape)
    assert far.any() and not out[far].any()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sigma,substeps", WIDE)
@pytest.mark.parametrize("at", [3, LONG // 2])
def test_large_value_spoils_no_small_ones(gpu, axis, sigma, substeps, at):
    """A voxel of 1 (at the low end, at the middle) on a background of 5e-7:
    away from it the error is relative to the background."""
    grid = GRIDS[axis]
    back = np.float32(5e-7)
    u = (back * (0.5 + vfd.synth_field(5, 0, 0, grid[::-1]))).astype(np.float32)
    u[(grid[2] // 2, grid[1] // 2, at) if axis == 0 else (grid[2] // 2, at, grid[0] // 2) if axis == 1 else
      (at, grid[1] // 2, grid[0] // 2)] = 1.0
    out, ref, mass = run_once(grid, u, sigma, substeps)
    assert rel_l2(out, ref) <= 2 * PER_GROUP
    far = np.broadcast_to(np.abs(along(axis, LONG) - at) > REACH, out.shape)
    assert far.any() and np.abs(out[far] - ref[far]).max() <= PER_GROUP * 1.5 * back


@pytest.mark.parametrize("sigma,substeps", [(1.4, 4), (2.6, 10)])
@pytest.mark.parametrize("kind", ["sparse", "signed"])
def test_sparse_and_signed_fields(gpu, sigma, substeps, kind):
    """Errors relative to what the products add up, sum |weight x value|: for
    a sparse field of positive values that is the output itself."""
    grid = (300, 70, 36)
    rng = np.random.default_rng(8)
    u = rng.standard_normal(grid[::-1])
    if kind == "sparse":
        u = np.where(rng.random(u.shape) < 0.02, np.exp(2.0 * u - 6.0), 0.0)
    u = u.astype(np.float32)
    out, ref, mass = run_once(grid, u, sigma, substeps)
    scale = oracle.tick(np.abs(u), sigma, 0.0, substeps, np.zeros(0, np.int32), np.zeros(0, np.float32))
    # the other axes' passes smooth |values| as far as values: the scale of the worst is the x pass'
    assert np.sqrt(((out - ref) ** 2).sum()) <= PER_GROUP * np.sqrt((scale ** 2).sum())


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_non_finite_values_reach_their_blocks_only(gpu, axis):
    grid = GRIDS[axis]
    u = vfd.synth_field(2, 0, 0, grid[::-1])
    bad = u.copy()
    bad[tuple(20 if a == 2 - axis else 1 for a in range(3))] = np.inf
    outs = []
    for v in (u, bad):
        with vfd.World(*grid, [vfd.field_params(0.6, 0.0)]) as w:
            w.upload(0, v)
            w.tick(1)
            outs.append(w.download(0))
    hit = ~np.isfinite(outs[1])
    assert hit[tuple(20 if a == 2 - axis else 1 for a in range(3))]
    assert not hit[np.broadcast_to(along(axis, LONG) > 20 + REACH, hit.shape)].any()
    np.testing.assert_array_equal(outs[0][~hit], outs[1][~hit])


@pytest.mark.parametrize("substeps", [1, 7])
def test_convolution_sum_next_to_a_baseline(gpu, substeps):
    """The accounting identity where the values hardly differ from the
    baseline: input, convolved and leaked sums are of the differences, so
    rounding the stored values (about the baseline) must not reach them."""
    nx, ny, nz, base = 132, 70, 35, 3e-4
    b = np.float32(base)
    u = (b * (1 + 1e-4 * np.random.default_rng(1).random((nz, ny, nx)))).astype(np.float32)
    with vfd.World(nx, ny, nz, [vfd.field_params(1.1, 0.0371, baseline=base)], pad_mode=vfd.PAD_CONSTANT_VF,
                   epi_boundary=125) as w:
        w.upload(0, u)
        w.tick(substeps)
        m, out = w.mass()[0], w.download(0)
    if substeps == 1:  # later substeps start from the decayed baseline, whose differences are not small
        v = np.zeros(u.shape)
        v[1:-1, 1:-1, 1:125] = u[1:-1, 1:-1, 1:125].astype(np.float64) - float(b)
        assert abs(m["input_sum"] - v.sum()) <= 1e-6 * v.sum()
    assert abs(m["input_sum"] - m["conv_sum"] - sum(m["leaked"])) <= 1e-6 * abs(m["input_sum"])
    assert abs(m["total"] - out.astype(np.float64).sum()) <= 1e-6 * abs(m["total"])


def test_wait_that_gave_up_reaches_its_own_world(gpu):
    """A banded pass's wait that gave up (run on purpose against a barrier that
    nothing completes, about 1 ms) is told once, by whichever synchronous call
    on its world comes next, and by no other world's; then the world ticks on."""
    grid, params = (40, 24, 16), [vfd.field_params(1.0, 0.1)]
    u = vfd.synth_field(1, 0, 0, grid[::-1])

    def gave_up(call):
        assert vfd.lib().vfd_world_check_wait(w._h, 2_000_000, None) == 0
        w.tick(2)  # later ticks do not clear the flag
        v.tick(2)
        assert v.mass()[0]["total"] > 0
        with pytest.raises(vfd.VfdError) as e:
            call()
        assert e.value.status == 5
        v.tick(2)
        call()

    with vfd.World(*grid, params) as w, vfd.World(*grid, params) as v:
        for x in (w, v):
            x.upload(0, u)
        out, d = [np.empty_like(u)], [np.zeros_like(u)]
        gave_up(w.mass)
        gave_up(lambda: w.diffuse_host([u], out, 2))
        gave_up(lambda: w.diffuse_update_host(out, d, np.ones(1, np.float32), 2))
        assert w.mass()[0]["total"] > 0


@pytest.mark.parametrize("what", ["world", "batch"])
@pytest.mark.parametrize("grid,sigma", [((90, 44, 31), 1.3), ((176, 160, 96), 0.9)])
def test_first_tick_captured(gpu, what, grid, sigma):
    """A fresh world's first tick of ten substeps under stream capture is the
    folded one (its operators are built beside the capture), and a replay
    gives what a direct tick gives."""
    import torch
    params = [vfd.field_params(sigma, 0.02)] * 2
    us = [vfd.synth_field(5, 0, f, grid[::-1]) for f in range(2)]
    with vfd.World(*grid, params) as w, vfd.World(*grid, params) as v:
        for f, u in enumerate(us):
            w.upload(f, u)
            v.upload(f, u)
        v.tick(10)
        v.tick(10)
        torch.cuda.synchronize()
        t = vfd.Batch([w]) if what == "batch" else w
        graph = torch.cuda.CUDAGraph()
        before = vfd.launch_count()
        with torch.cuda.graph(graph):
            t.tick(10, stream=torch.cuda.current_stream().cuda_stream)
        # three operators' set-up kernels, three passes, and a batch's accounting reset
        assert vfd.launch_count() - before <= 7
        torch.cuda.synchronize()
        for f, u in enumerate(us):
            np.testing.assert_array_equal(w.download(f), u)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        for f in range(2):
            np.testing.assert_array_equal(w.download(f), v.download(f))
        del graph
        if what == "batch":
            t.close()


def test_operators_are_ready_on_every_stream(gpu):
    """Operators are built on a stream of their own: a first tick on one stream
    and the next on another, right after, use them complete."""
    import torch
    grid, params = (200, 60, 50), [vfd.field_params(1.3 + 0.1 * f, 0.02) for f in range(4)]
    us = [vfd.synth_field(6, 0, f, grid[::-1]) for f in range(4)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for k in range(3):
        with vfd.World(*grid, params) as w, vfd.World(*grid, params) as v:
            for x in (w, v):
                for f, u in enumerate(us):
                    x.upload(f, u)
            torch.cuda.synchronize()
            if k < 2:
                for m in (2 + k, 9):
                    w.tick(m, stream=streams[0].cuda_stream)
                    v.tick(m, stream=streams[1].cuda_stream)
            else:
                with vfd.Batch([w, v]) as b:
                    b.tick(2, stream=streams[0].cuda_stream)
                    b.tick(9, stream=streams[1].cuda_stream)
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            outs.append([x.download(f) for x in (w, v) for f in range(4)])
    for f in range(4):
        np.testing.assert_array_equal(outs[0][f], outs[0][4 + f])
        np.testing.assert_array_equal(outs[0][f], outs[2][f])
        np.testing.assert_array_equal(outs[1][f], outs[1][4 + f])


def test_operators_are_built_for_ticks_that_use_them(gpu):
    """A large world of narrow kernels runs single substeps on the FFT passes:
    it holds no banded operators until a tick of several substeps."""
    grid, params = (256, 160, 128), [vfd.field_params(0.9, 0.02)] * 2
    vfd.autotune_clear()
    try:
        with vfd.World(*grid, params) as w:
            w.tick(1)
            single = w.device_bytes()
            w.tick(10)
            assert w.device_bytes() > single
        vfd.autotune_set(*grid, params, [{"method": "register_fft"}] * 3)
        with vfd.World(*grid, params) as w:  # no banded products at all
            w.tick(1)
            assert w.device_bytes() == single
    finally:
        vfd.autotune_clear()


def test_batch_alternates_substep_counts(gpu):
    """Ticks of one and of several substeps in turn, over worlds that take the
    FFT passes always (pinned), for single substeps (large, narrow kernels) and
    never: every tick equals the world's own."""
    vfd.autotune_clear()
    try:
        vfd.autotune_set(44, 40, 36, [vfd.field_params(1.0, 0.02)] * 2, [{"method": "register_fft"}] * 3)
        specs = [((44, 40, 36), 1.0), ((176, 160, 96), 0.9), ((90, 33, 70), 2.6)]
        worlds, singles = [], []
        for i, (g, sig) in enumerate(specs):
            for out in (worlds, singles):
                w = vfd.World(*g, [vfd.field_params(sig, 0.02)] * 2)
                for f in range(2):
                    w.upload(f, vfd.synth_field(3, i, f, g[::-1]))
                out.append(w)
        with vfd.Batch(worlds) as b:
            for n in (1, 4, 1, 4, 4, 4, 1, 1, 1, 6, 1):
                b.tick(n)
                for w, v in zip(worlds, singles):
                    v.tick(n)
                    for f in range(2):
                        np.testing.assert_array_equal(w.download(f), v.download(f))
        for w in worlds + singles:
            w.close()
    finally:
        vfd.autotune_clear()


def test_batch_of_many_fields(gpu):
    """More than 65535 fields in one batch."""
    grid, nf, n = (4, 3, 2), 1200, 56
    params = [vfd.field_params(0.5, 0.02)] * nf
    worlds = [vfd.World(*grid, params) for _ in range(n)]
    u = [vfd.synth_field(7, 0, f, grid[::-1]) for f in range(4)]
    probe = [(0, 0), (n // 2, 5), (n - 1, nf - 1), (n - 2, 17)]
    for k, (i, f) in enumerate(probe):
        worlds[i].upload(f, u[k])
    with vfd.Batch(worlds) as b:
        b.tick(2)
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    for k, (i, f) in enumerate(probe):
        assert rel_l2(worlds[i].download(f), oracle.tick(u[k], 0.5, 0.02, 2, *none)) <= PER_GROUP
    assert not worlds[1].download(3).any()
    for w in worlds:
        w.close()


@pytest.mark.parametrize("what", ["world", "batch"])
@pytest.mark.parametrize("when", ["before", "after"])
@pytest.mark.parametrize("grid,sigma", [((90, 44, 31), 1.3), ((176, 160, 96), 0.9)])
def test_no_memory_for_operators(gpu, monkeypatch, what, when, grid, sigma):
    """Operators that find no memory (a bound of one byte, before or after the
    world is created) leave ticks on what the world was created with."""
    nf = 2
    params = [vfd.field_params(sigma, 0.02)] * nf
    us = [vfd.synth_field(5, 0, f, grid[::-1]) for f in range(nf)]
    if when == "before":
        monkeypatch.setenv("VFD_BAND_BYTES", "1")
    with vfd.World(*grid, params) as w:
        monkeypatch.setenv("VFD_BAND_BYTES", "1")
        for f, u in enumerate(us):
            w.upload(f, u)
        t = vfd.Batch([w]) if what == "batch" else w
        for n in (4, 1, 4):
            t.tick(n)
        got = [w.download(f) for f in range(nf)]
        mass = w.mass()
        if what == "batch":
            t.close()
    none = (np.zeros(0, np.int32), np.zeros(0, np.float32))
    for f, u in enumerate(us):
        ref = oracle.tick(u, sigma, 0.02, 9, *none)
        assert rel_l2(got[f], ref) <= 1e-5
        assert abs(mass[f]["total"] - ref.sum()) <= 1e-5 * ref.sum()


def test_device_memory_is_accounted(gpu):
    """vfd_world_device_bytes tells what a world's passes hold by then, and a
    server counts the operators of its ticks' substeps against its budget."""
    grid, params, nf = (176, 160, 96), [vfd.field_params(0.9, 0.02)] * 4, 4
    fields = 4 * nf * int(np.prod(grid))
    with vfd.World(*grid, params) as w:  # FFT passes: jobs, tiles, tensor maps
        fft = w.device_bytes() - fields
        w.tick(10)
        both = w.device_bytes() - fields
    small = (64, 64, 32)
    with vfd.World(*small, params) as w:  # banded products alone
        one = w.device_bytes() - 4 * nf * int(np.prod(small))
        w.tick(10)
        ten = w.device_bytes()
    # an axis' operator holds at least one image of 5 (one substep of radius 3) or
    # 8 (ten) k-steps of 6 KB, the tiles of the FFT passes 16 bytes each
    assert one >= 3 * nf * 5 * 6144 and both - fft >= 3 * nf * 8 * 6144
    assert fft >= sum(16 * nf * (np.prod(grid) // n // 32) for n in grid) // 4
    with vfd.Server(8 << 30, max_active=2, substeps_per_tick=10) as s:
        rid = s.submit(small, params, 3, synth=(7, 0, 0.0, 1e-3))
        assert s.wait(rid)["status"] == 0
        assert s.stats()["hbm_peak"] >= ten


@pytest.mark.parametrize("scale", [1e-33, 1e-20, 1.0, 1e20, 1e36])
@pytest.mark.parametrize("substeps", [1, 6])
def test_scales(gpu, scale, substeps):
    """Positive fields over FP32's range (from 2^-110 on, where the third part
    of a value underflows, to where a block's sum overflows)."""
    grid = (140, 33, 41)
    u = ((0.2 + np.random.default_rng(3).random(grid[::-1])) * scale).astype(np.float32)
    out, ref, mass = run_once(grid, u, 1.4, substeps)
    assert rel_l2(out / scale, ref / scale) <= PER_GROUP
