"""Calls whose expert kernel is the tcgen05 fold kernel, bit for bit against the CPU oracle: single matrices,
expert groups, layers and wide shared experts, at the edges of its tiles and of the rules that choose it."""
import ctypes as C

import numpy as np
import pytest

import oracle as po
from peregrine_b200 import cuda
from peregrine_b200.resident import upload_layer
from peregrine_b200.synth import synth_expert, synth_layer, synth_matrix, synth_tokens
from tests import hostcheck as hc
from tests.gpu_common import bits
from tests.refmodel import oracle_layer_forward

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
    k, rows = 2048, 5000
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
    pick = np.r_[0:40, 2480:2520, rows - 40:rows]
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
