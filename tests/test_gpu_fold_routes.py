"""Calls whose expert kernel is the tcgen05 fold kernel, bit for bit against the CPU oracle: single matrices,
expert groups, layers and wide shared experts, at the edges of its tiles and of the rules that choose it."""
import ctypes as C

import numpy as np
import pytest

import oracle as po
from peregrine_b200 import cuda
from peregrine_b200.resident import upload_expert, upload_layer
from peregrine_b200.synth import synth_expert, synth_layer, synth_matrix, synth_tokens
from tests import hostcheck as hc
from tests.gpu_common import bits
from tests.refmodel import o_expert, oracle_layer_forward

pytestmark = pytest.mark.gpu


def upload(dev, m):
    return (cuda.Tensor.upload_grouped(dev, m.q, m.scale, m.i_n, m.o_n, m.gs) if m.gs
            else cuda.Tensor.upload(dev, m.q, m.scale, 2, m.i_n, m.o_n))


def apply(m, x):
    return po.Weight(m.q, m.scale, 4 if m.gs else 2, m.gs, m.i_n, m.o_n).apply(x, x.shape[0])


class DevRows:
    def __init__(self, dev, rows, width):
        self.dev, self.shape = dev, (rows, width)
        self.ptr = cuda.lib().coli_cuda_pipe_alloc(dev, rows * width * 4)
        assert self.ptr

    def put(self, a):
        a = np.ascontiguousarray(a, np.float32)
        assert cuda.lib().coli_cuda_pipe_upload(self.dev, self.ptr, a.ctypes.data, a.nbytes) == 1

    def get(self, rows=None):
        out = np.empty((self.shape[0] if rows is None else rows, self.shape[1]), np.float32)
        assert cuda.lib().coli_cuda_pipe_download(self.dev, self.ptr, out.ctypes.data, out.nbytes) == 1
        return out

    def free(self):
        cuda.lib().coli_cuda_pipe_free(self.dev, self.ptr)


def fold_launches(dev, call):
    """Runs `call` and returns its result and how many of its launches were the fold kernel's (None where the
    profiler records no kernels)."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = call()
        assert cuda.lib().coli_cuda_pipe_sync(dev) == 1
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "kernel" in e.name]
    return out, sum("ffn_w4a8_fold_kernel" in n for n in names) if names else None


def gemm(t, y, x, rows):
    return cuda.lib().coli_cuda_pipe_gemm(t.handle, C.c_void_p(y.ptr), C.c_void_p(x.ptr), rows)


def test_scratch_depends_on_rows_and_width_not_on_the_kernel(dev):
    """A call that has sized the scratch for its rows and width has sized it for every matrix of that width: the
    product of a taller one, which the fold kernel takes, is recorded without a call of its own before (growing
    scratch would end the recording), and the replay gives the oracle's rows.  The row count is above all others
    of the suite, so that no earlier test has left more scratch behind."""
    lib = cuda.lib()
    rng = np.random.default_rng(61)
    k, rows = 2048, 4500
    assert not hc.fold_beats_block(200, k, 32, 1, rows) and hc.fold_beats_block(600, k, 32, 1, rows)
    small, tall = synth_matrix(rng, 200, k, 32), synth_matrix(rng, 600, k, 32)
    ts, tt = upload(dev, small), upload(dev, tall)
    x, y = DevRows(dev, rows, k), DevRows(dev, rows, 600)
    xh = rng.standard_normal((rows, k)).astype(np.float32)
    x.put(xh)
    assert gemm(ts, y, x, rows) == 1 and lib.coli_cuda_pipe_sync(dev) == 1
    assert lib.coli_cuda_graph_begin(dev) == 1
    rc = gemm(tt, y, x, rows)
    g = C.c_void_p()
    assert lib.coli_cuda_graph_end(dev, C.byref(g)) == 1 and rc == 1
    assert lib.coli_cuda_graph_launch(g) == 1
    pick = np.r_[0:40, 2240:2280, rows - 40:rows]
    assert np.array_equal(bits(y.get()[pick]), bits(apply(tall, xh[pick])))
    assert cuda.last_device_error(dev) == 0
    lib.coli_cuda_graph_free(g)
    for b in (x, y, ts, tt):
        b.free()


@pytest.mark.parametrize("m,want_fold", [(300, 1), (650, 2)])
def test_wide_shared_expert_chooses_per_phase(dev, m, want_fold):
    """A shared expert of its own width: 300 tokens fill the SMs with gate/up items (20 weight blocks) but not
    with down items (8), 650 tokens with both."""
    hidden, wide = 2048, 2560
    assert hc.fold_beats_block(wide, hidden, 32, 0, m)
    assert hc.fold_beats_block(hidden, wide, 32, 1, m) == (want_fold == 2)
    layer = synth_layer(31, hidden=hidden, inter=256, n_experts=24, k=1, gs=32, distinct_experts=2)
    layer.shared = synth_expert(np.random.default_rng(310), hidden, wide, 32)
    ml = upload_layer(dev, layer)
    x = synth_tokens(32, m, hidden)
    out = np.empty_like(x)
    ml.forward(x, out)  # sizes the scratch
    got, n = fold_launches(dev, lambda: ml.forward(x, out))
    if n is not None:
        assert n == want_fold + routed_folds(layer, m)
    assert np.array_equal(bits(got), bits(oracle_layer_forward(layer, x, threads=8)))
    assert cuda.last_device_error(dev) == 0
    ml.free()


def routed_folds(layer, m):
    """Launches of the routed experts that go to the fold kernel."""
    return hc.layer_route(layer.hidden, layer.inter, layer.gs, m, layer.n_experts, layer.k).count("fold")


@pytest.mark.parametrize("hidden,inter,m,experts,k,want", [
    (2048, 256, 160, 100, 2, ("fold", "tiles")),   # one chunk of inter
    (1024, 2048, 300, 36, 4, ("tiles", "fold")),   # four chunks of hidden
])
def test_layer_phases_on_different_kernels(dev, hidden, inter, m, experts, k, want):
    assert hc.layer_route(hidden, inter, 0, m, experts, k) == want
    layer = synth_layer(90 + k, hidden=hidden, inter=inter, n_experts=experts, k=k, gs=0, distinct_experts=3)
    ml = upload_layer(dev, layer)
    x = synth_tokens(91, m, hidden)
    out = np.empty_like(x)
    ml.forward(x, out)
    got, n = fold_launches(dev, lambda: ml.forward(x, out))
    assert n is None or n == 1
    assert np.array_equal(bits(got), bits(oracle_layer_forward(layer, x, threads=8)))
    assert cuda.last_device_error(dev) == 0
    ml.free()


def test_layer_with_few_items_stays_with_the_tiles(dev):
    """Eight experts of 2048 x 256 give the fold kernel 18 gate/up items for 148 SMs (us: 35 with the tiles, 51)."""
    layer = synth_layer(95, hidden=2048, inter=256, n_experts=8, k=2, gs=32, distinct_experts=2)
    ml = upload_layer(dev, layer)
    x = synth_tokens(96, 64, 2048)
    ml.forward(x)
    got, n = fold_launches(dev, lambda: ml.forward(x))
    assert n is None or n == 0
    assert np.array_equal(bits(got), bits(oracle_layer_forward(layer, x, threads=8)))
    ml.free()


def test_fold_rows_take_no_scratch_of_their_own(dev):
    """A layer's scratch for 8192 tokens is what the int8 layouts need, also where both phases take the fold kernel:
    its fp16 rows lie in buffers that are idle at the time (their own would be 212 MB here)."""
    import torch

    hidden, inter, experts, k = 2048, 1024, 16, 8

    def scratch(m):
        pairs, kp, kpd = m * (k + 1), hidden, inter
        return (pairs * (kp + kpd) * 17 // 16 + pairs * (kp + kpd) // 8 + pairs * 4 * (hidden + inter + 5)
                + m * (kp + kp // 8 + hidden * 4 * 260 // 256 + 4 * experts + 16 * k))

    layer = synth_layer(97, hidden=hidden, inter=inter, n_experts=experts, k=k, gs=32, distinct_experts=1)
    ml = upload_layer(dev, layer, repeats="clone")
    x = torch.randn(8192, hidden, device="cuda")
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    free = []
    for m in (512, 8192):
        assert hc.layer_route(hidden, inter, 32, m, experts, k) == ("fold", "fold")
        ml.forward_dev(out.data_ptr(), x.data_ptr(), m)
        assert cuda.lib().coli_cuda_pipe_sync(dev) == 1
        free.append(cuda.mem_info(dev)[0])
    grown, want = free[0] - free[1], scratch(8192) - scratch(512)
    assert want - (64 << 20) < grown < want + (64 << 20), (grown, want)
    ml.free()


def same(got, want):
    """Equal bits; NaNs (whose payload no rule fixes) in the same places."""
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(bits(got)[~nan], bits(want)[~nan])


@pytest.mark.parametrize("gs", [0, 32, 64, 128, 256])
def test_one_matrix(dev, gs):
    """32 to 127 rows: one and two column halves, one and two row blocks; ragged K and O; rows of zeros, with an
    infinity and with a NaN."""
    rng = np.random.default_rng(300 + gs)
    k, o = 2041, 33003  # 8 chunks, the last short by 7 elements; the last weight block holds 235 rows
    assert all(hc.fold_beats_block(o, k, gs, 1, s) for s in (33, 64, 100, 127))
    m = synth_matrix(rng, o, k, gs)
    t = upload(dev, m)
    x, y = DevRows(dev, 127, k), DevRows(dev, 127, o)
    xh = rng.standard_normal((127, k)).astype(np.float32)
    xh[5] = 0.0
    xh[6, 3] = np.inf   # the row's scale is infinite, its codes are zero
    xh[7, 11] = np.nan  # never the maximum; its code is zero
    x.put(xh)
    want = apply(m, xh)
    for rows in (32, 33, 64, 65, 100, 127):
        assert gemm(t, y, x, rows) == 1
        assert same(y.get(rows), want[:rows]), rows
    assert cuda.last_device_error(dev) == 0
    for b in (x, y, t):
        b.free()


def test_one_matrix_recorded(dev):
    """A product of the fold kernel inside a recorded graph (its tensor map travels with the kernel's arguments),
    replayed with x changed in place."""
    lib = cuda.lib()
    rng = np.random.default_rng(44)
    k, o, rows = 2048, 33003, 64
    assert hc.fold_beats_block(o, k, 32, 1, rows)
    m = synth_matrix(rng, o, k, 32)
    t = upload(dev, m)
    xs = [rng.standard_normal((rows, k)).astype(np.float32) for _ in range(3)]
    x, y = DevRows(dev, rows, k), DevRows(dev, rows, o)
    x.put(xs[0])
    assert gemm(t, y, x, rows) == 1 and lib.coli_cuda_pipe_sync(dev) == 1
    assert lib.coli_cuda_graph_begin(dev) == 1
    rc = gemm(t, y, x, rows)
    g = C.c_void_p()
    assert lib.coli_cuda_graph_end(dev, C.byref(g)) == 1 and rc == 1
    for xh in xs[1:]:
        x.put(xh)
        assert lib.coli_cuda_graph_launch(g) == 1
        assert np.array_equal(bits(y.get()), bits(apply(m, xh)))
    lib.coli_cuda_graph_free(g)
    for b in (x, y, t):
        b.free()


def test_per_row_scales_at_the_largest_exact_row(dev):
    """Per-row scales: the fp32 accumulator holds the dot of the whole row.  K = 16384 is the longest row the
    kernel is given (8 * 127 * 16384 < 2^24); all codes at their extremes, alternating signs and odd dots reach
    the largest sums and the smallest differences of large sums.  One more element goes to another kernel."""
    rng = np.random.default_rng(16)
    o = 14096
    assert hc.fold_beats_block(o, 16384, 0, 1, 33) and not hc.fold_beats_block(o, 16385, 0, 1, 33)
    for k in (16384, 16385):
        m = synth_matrix(rng, o, k, 0)
        q = m.q.reshape(o, -1)
        q[0] = 0x00                     # -8, -8, ..
        q[1] = 0xFF                     # +7, +7, ..
        q[2], q[2, ::2] = 0x00, 0xFF
        q[3], q[3, :q.shape[1] // 2] = 0xFF, 0x00
        q[4], q[4, -1] = 0x00, 0x01     # -8 .., the last but one (K odd: the last) code -7
        if k % 2:
            q[:, -1] &= 0x0F
        t = upload(dev, m)
        xh = rng.standard_normal((33, k)).astype(np.float32)
        xh[0], xh[1] = 1.0, -1.0
        xh[2] = 1.0
        xh[2, ::2] = -1.0
        xh[3] = 0.0                     # every product is a zero, some of them negative
        xh[4] = np.where(np.arange(k) % 3 == 0, 1.0, 126.0 / 127.0)
        x, y = DevRows(dev, 33, k), DevRows(dev, 33, o)
        x.put(xh)
        assert gemm(t, y, x, 33) == 1
        got = y.get()
        pick = np.r_[0:64, o - 64:o]
        part = type(m)(np.ascontiguousarray(q[pick]).reshape(-1), m.scale[pick], k, pick.size, 0)
        assert np.array_equal(bits(got[:, pick]), bits(apply(part, xh))), k
        for b in (x, y, t):
            b.free()
    assert cuda.last_device_error(dev) == 0


@pytest.mark.parametrize("hidden,inter,gs,rows", [
    (2048, 1024, 0, [1, 120] + [(7 * i) % 121 + 1 for i in range(14)]),    # gate/up folds, down (4 chunks) does not
    (2048, 1024, 128, [1, 120] + [(7 * i) % 121 + 1 for i in range(14)]),
    (2056, 2056, 32, [64] * 8 + [63, 33, 1, 64]),                          # both fold, 9 chunks, ragged K and O
])
def test_expert_group(dev, hidden, inter, gs, rows):
    rng = np.random.default_rng(700 + gs)
    want_fold = hc.fold_beats_block(inter, hidden, gs, 0, rows) + hc.fold_beats_block(hidden, inter, gs, 1, rows)
    assert want_fold == (2 if inter > 2048 else 1)
    kinds = [synth_expert(rng, hidden, inter, gs) for _ in range(3)]
    up = [upload_expert(dev, e, hidden, inter) for e in kinds]
    n = len(rows)
    x = rng.standard_normal((sum(rows), hidden)).astype(np.float32)
    gpu = [up[i % 3] for i in range(n)]
    want, at = [], 0
    for i, r in enumerate(rows):
        want.append(po.swiglu(*o_expert(kinds[i % 3]), x[at:at + r], r))
        at += r
    want = np.concatenate(want)
    cuda.expert_group(gpu, rows, x, hidden)
    got, folds = fold_launches(dev, lambda: cuda.expert_group(gpu, rows, x, hidden))
    assert folds is None or folds == want_fold
    assert np.array_equal(bits(got), bits(want))
    # the reduce form: every row added to one of 50 tokens, in row order
    dst = np.arange(sum(rows)) % 50
    rw = rng.random(sum(rows)).astype(np.float32)
    red = cuda.expert_group_reduce(gpu, rows, x, hidden, cuda.ReduceLayout.build(dst, 50), rw, 50)
    acc = np.zeros((50, hidden), np.float32)
    for j, d in enumerate(dst):
        acc[d] = acc[d] + (rw[j] * want[j]).astype(np.float32)
    assert np.array_equal(bits(red), bits(acc))
    assert cuda.last_device_error(dev) == 0
    for e in up:
        e.free()


@pytest.mark.parametrize("gs,hidden,inter,m", [(256, 2304, 520, 70), (256, 300, 256, 3), (0, 1000, 264, 65)])
def test_forced_layers(dev, monkeypatch, gs, hidden, inter, m):
    """Groups of 256 (one group a chunk), per-row scales over several chunks, inter and hidden off every tile."""
    monkeypatch.setenv("PEREGRINE_B200_TILE", "2")
    layer = synth_layer(800 + m, hidden=hidden, inter=inter, n_experts=6, k=2, gs=gs)
    x = synth_tokens(81, m, hidden)
    ml = upload_layer(dev, layer)
    ml.forward(x)
    got, n = fold_launches(dev, lambda: ml.forward(x))
    assert n is None or n == 2
    assert np.array_equal(bits(got), bits(oracle_layer_forward(layer, x, threads=8)))
    assert cuda.last_device_error(dev) == 0
    ml.free()
