"""The tensor-core path of factorable tables (code_gemm, AMSIM_CODES=1 forces it at any size) against
deterministic mode, which is bit-identical to the reference: every table factorisation (32, 64 and 128
slots), every operand layout the kernel fetches, and the sizes where its tiles and stages end.

Bound: products are exact; an accumulator takes at most 128 steps (256 instructions with 128 slots) and each
truncates by less than 2^-23 of a partial sum, half of that on average: at most 256 * 2^-24 = 1.5e-5 of the largest
partial sum if every instruction lost bits.  A product has at most 9 significant bits, so with ordinary operands few
do; with widely spread exponents nearly all do, on sums that grow over the chunk (the factor 1/2 of a mean):
1e-5 as for every fast kernel.  test_no_further_from_64_bits compares both paths with exact sums."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import lut_path, rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def forced(monkeypatch):
    from approxtrain_b200 import _lib
    monkeypatch.setenv("AMSIM_CODES", "1")
    _lib.lib.amsim_debug_reload_env()
    yield _lib
    stuck = C.c_uint(1)
    assert _lib.lib.amsim_debug_wait_report(C.byref(stuck)) == 0 and stuck.value == 0, "a wait between warps ran out"
    monkeypatch.undo()
    _lib.lib.amsim_debug_reload_env()


def _close(got, want):
    assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5


# (n, h, w, c, kh, kw, k, stride, padding): tile edges in pixels and channels (k 64 / 65 / 128 / 129 / 257), taps that
# end inside a 16-step block (c 8, 24, 37), reductions of one block, of more than one 128-step chunk, strides
SHAPES = [(1, 16, 16, 16, 1, 1, 64, 1, "VALID"), (2, 9, 13, 16, 3, 3, 65, 1, "SAME"), (1, 16, 16, 24, 3, 3, 128, 1, "SAME"),
          (3, 11, 7, 8, 3, 3, 129, 2, "SAME"), (2, 12, 12, 37, 5, 5, 257, 1, "SAME"), (1, 30, 30, 3, 7, 7, 64, 2, "VALID"),
          (2, 14, 14, 256, 1, 1, 300, 1, "VALID"), (4, 20, 20, 64, 3, 3, 32, 1, "SAME")]


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MIT_5", "ACC_7", "MBM_1"])
@pytest.mark.parametrize("shape", SHAPES)
def test_convolutions(forced, lut, shape):
    from approxtrain_b200 import ops
    n, h, w, c, kh, kw, k, s, pad = shape
    g = torch.Generator(device="cuda").manual_seed(n * h + k)
    x = torch.relu(torch.randn(n, h, w, c, generator=g, device="cuda"))
    wt = torch.randn(kh, kw, c, k, generator=g, device="cuda")
    kw_ = dict(strides=s, padding=pad, mant_mul_lut=lut_path(lut))
    y = ops.convam(x, wt, **kw_)
    _close(y, ops.convam(x, wt, deterministic=True, **kw_))
    assert torch.equal(y, ops.convam(x, wt, **kw_)), "run-to-run identical"
    dy = torch.randn(y.shape, generator=g, device="cuda")
    _close(ops.convam_input_grad(x.shape, wt, dy, **kw_), ops.convam_input_grad(x.shape, wt, dy, deterministic=True, **kw_))
    dw = ops.convam_filter_grad(wt.shape, x, dy, **kw_)
    _close(dw, ops.convam_filter_grad(wt.shape, x, dy, deterministic=True, **kw_))
    assert torch.equal(dw, ops.convam_filter_grad(wt.shape, x, dy, **kw_)), "run-to-run identical"


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MBM_5"])
@pytest.mark.parametrize("m,k,n,ta,tb", [(128, 64, 128, 0, 1), (100, 70, 90, 1, 0), (33, 129, 257, 1, 1), (128, 128, 64, 0, 0), (1, 5, 1, 0, 0)])
def test_matmuls(forced, lut, m, k, n, ta, tb):
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a = torch.randn(*((3, k, m) if ta else (3, m, k)), generator=g, device="cuda")
    b = torch.randn(*((3, n, k) if tb else (3, k, n)), generator=g, device="cuda")
    f = lambda det: ops.matmulam(a, b, transpose_a=bool(ta), transpose_b=bool(tb), mant_mul_lut=lut_path(lut),  # noqa: E731
                                 deterministic=det, alpha=0.125)
    _close(f(False), f(True))


def _on(forced, codes, f):
    os.environ["AMSIM_CODES"] = str(codes)
    forced.lib.amsim_debug_reload_env()
    return f()


def _same_as_table_kernels(forced, f):
    """Not finite where the table kernels' result is not, in the same way, and close elsewhere."""
    got, want = _on(forced, 1, f), _on(forced, 0, f)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    finite = torch.isfinite(want)
    assert finite.any()
    _close(got[finite], want[finite])


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MIT_5", "MBM_5"])
@pytest.mark.parametrize("e", [121, 123, 125, 127])
def test_products_up_to_the_largest_float(forced, lut, e):
    """Products of 2^e and their cancelling sums: FP32 holds them, accumulators in units of the table's step do not."""
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(e)
    x, w = torch.randn(300, 130, generator=g, device="cuda"), torch.randn(130, 200, generator=g, device="cuda")
    big = 2.0 ** (e // 2)
    x[5:40, 7], w[7, 3:90] = 2.0 ** (e - e // 2), big
    _same_as_table_kernels(forced, lambda: ops.denseam(x, w, lut_path(lut)))
    w[3, 3:90], x[5:40, 3] = -big, 2.0 ** (e - e // 2)      # the sum returns to ordinary size
    f = lambda: ops.denseam(x, w, lut_path(lut))  # noqa: E731
    got, want = _on(forced, 1, f), _on(forced, 0, f)
    assert torch.isfinite(want).all() and torch.isfinite(got).all()
    # 130 additions in any order, each off by at most 2^-23 of a partial sum of about 2^e
    assert (got[5:40, 3:90].double() - want[5:40, 3:90]).abs().max() <= 130 * 2.0 ** (e - 22)
    other = torch.ones_like(got, dtype=torch.bool)
    other[5:40, 3:90] = False
    _close(got[other], want[other])


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7"])
@pytest.mark.parametrize("shape", [(2, 9, 13, 16, 3, 3, 65, 1, "SAME"), (3, 11, 7, 8, 3, 3, 129, 2, "SAME"), (1, 30, 30, 3, 7, 7, 64, 2, "VALID"),
                                   (2, 14, 14, 64, 1, 1, 300, 1, "VALID")])
def test_huge_operands_in_every_direction(forced, lut, shape):
    """Sums between 2^122 and 2^128, and products beyond."""
    from approxtrain_b200 import ops
    n, h, w, c, kh, kw, k, s, pad = shape
    g = torch.Generator(device="cuda").manual_seed(h + k)
    kw_ = dict(strides=s, padding=pad, mant_mul_lut=lut_path(lut))
    x, wt = torch.randn(n, h, w, c, generator=g, device="cuda"), torch.randn(kh, kw, c, k, generator=g, device="cuda")
    x[0, 3, 4, 1], x[0, 5, 5, 2], x[n - 1, 6, 2, 0] = 2.0 ** 100, -2.0 ** 62, 2.0 ** 63
    wt[0, 0, 1, 5], wt[0, 0, 2, 9], wt[kh - 1, 0, 0, 7] = 2.0 ** 25, 2.0 ** 63, -2.0 ** 61
    _same_as_table_kernels(forced, lambda: ops.convam(x, wt, **kw_))
    b, sc = torch.randn(k, generator=g, device="cuda"), torch.rand(k, generator=g, device="cuda") - 0.5
    _same_as_table_kernels(forced, lambda: ops.convam_bias_act(x, wt, b, activation="relu", scale=sc, **kw_))
    dy = torch.randn(ops.convam(x, wt, **kw_).shape, generator=g, device="cuda")
    dy[0, 2, 1, 5], dy[0, 1, 2, 9], dy[0, 3, 3, 7] = 2.0 ** 99, 2.0 ** 61, 2.0 ** 62
    _same_as_table_kernels(forced, lambda: ops.convam_input_grad(x.shape, wt, dy, **kw_))
    _same_as_table_kernels(forced, lambda: ops.convam_filter_grad(wt.shape, x, dy, **kw_))
    if kh == 1:
        a, b = x[0, :, :, :].reshape(-1, c).t().contiguous(), wt[0, 0]
        _same_as_table_kernels(forced, lambda: ops.matmulam(a, b, transpose_a=True, alpha=0.5, mant_mul_lut=lut_path(lut)))


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7"])
def test_a_non_finite_operand_makes_its_outputs_nan_and_no_others(forced, lut):
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(9)
    x, w = torch.randn(700, 300, generator=g, device="cuda"), torch.randn(300, 200, generator=g, device="cuda")
    clean = ops.denseam(x, w, lut_path(lut))
    x[3, 7], x[600, 299], w[5, 11], w[6, 190] = float("inf"), float("nan"), -float("inf"), float("nan")
    y = ops.denseam(x, w, lut_path(lut))
    bad = torch.zeros(700, 200, dtype=torch.bool, device="cuda")
    bad[3], bad[600], bad[:, 11], bad[:, 190] = True, True, True, True
    assert torch.equal(torch.isnan(y), bad) and torch.equal(y[~bad], clean[~bad])


def _exact_gemm(a, b, lut):
    """sum_k AM(a[i, k], b[k, j]) in 64 bits, products from the elementwise op."""
    from approxtrain_b200 import ops
    m = int(lut.split("_")[1])
    s = 1 + torch.arange(1 << m, device="cuda") / float(1 << m)
    table = ops.am_multiply(s[:, None].expand(1 << m, 1 << m).contiguous(), s[None, :].expand(1 << m, 1 << m).contiguous(),
                            lut_path(lut)).double().flatten()

    def split(x):
        bits = x.contiguous().view(torch.int32)
        e = (bits >> 23) & 255
        scale = torch.ldexp(torch.where(bits < 0, -1.0, 1.0).double(), (e - 127).double())
        return torch.where(e > 0, scale, torch.zeros_like(scale)), ((bits >> (23 - m)) & ((1 << m) - 1)).long()
    (sa, ia), (sb, ib) = split(a), split(b)
    out = torch.zeros(a.shape[0], b.shape[1], dtype=torch.float64, device="cuda")
    for k in range(a.shape[1]):
        out += table[ia[:, k, None] * (1 << m) + ib[None, k]] * (sa[:, k, None] * sb[None, k])
    return out


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MIT_5"])
@pytest.mark.parametrize("data", ["activations", "normal", "positive", "spread"])
@pytest.mark.parametrize("k,q", [(64, 256), (147, 64), (256, 256), (512, 300), (576, 64), (1152, 128), (2304, 256)])
def test_no_further_from_64_bits(forced, lut, data, k, q):
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(k)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w = r(512, k), r(k, q)
    if data == "activations":
        x, w = torch.relu(x), w * (2.0 / k) ** 0.5
    elif data == "positive":
        x, w = torch.rand(512, k, generator=g, device="cuda"), torch.rand(k, q, generator=g, device="cuda")
    elif data == "spread":
        x, w = (t * 2.0 ** torch.randint(-10, 11, t.shape, generator=g, device="cuda") for t in (x, w))
    want = _exact_gemm(x, w, lut)
    err = lambda y: float((y.double() - want).norm() / want.norm())  # noqa: E731
    here, table = err(_on(forced, 1, lambda: ops.denseam(x, w, lut_path(lut)))), err(_on(forced, 0, lambda: ops.denseam(x, w, lut_path(lut))))
    if data == "spread":
        assert here <= 1e-5 / 2      # nearly every instruction truncates: half of 256 * 2^-24, on half the final sum
    elif k < (64 if lut == "MBM_7" else 128):
        pass                         # such reductions take this path only when it is forced
    else:
        # as close as the table kernels; few of the outputs are off at all in short reductions, so the two figures
        # scatter by a tenth from seed to seed
        assert here <= 1.2 * table, (here, table)


def test_zeros_give_zero_and_non_finite_values_stay_visible(forced):
    from approxtrain_b200 import ops
    p = lut_path("MBM_7")
    x = torch.zeros(200, 64, device="cuda")
    w = torch.randn(64, 96, device="cuda")
    assert torch.equal(ops.denseam(x, w, p), torch.zeros(200, 96, device="cuda"))
    x[7, 3] = float("nan")
    y = ops.denseam(x, w, p)
    assert not torch.isfinite(y[7]).any() and torch.equal(y[:7], torch.zeros(7, 96, device="cuda"))


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MIT_5"])
@pytest.mark.parametrize("rows,width,units", [(64, 4096, 4096), (100, 2048, 2050), (862, 925, 256), (900, 931, 250), (6272, 256, 1024)])
def test_the_queried_workspace_serves_whatever_plan_is_taken(lut, rows, width, units):
    """A launch that is handed more than the query asks for takes the same plan: the same bits."""
    from approxtrain_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, dy = torch.randn(rows, width, generator=g, device="cuda"), torch.randn(rows, units, generator=g, device="cuda")
    need = _lib.lib.amsim_dense_bwd_weight_workspace(rows, units, width, 0)

    def grad(extra):
        ws, dw = torch.empty(need + extra, dtype=torch.uint8, device="cuda"), torch.empty(width, units, device="cuda")
        _lib.check(_lib.lib.amsim_dense_bwd_weight(ops._stream(), ops.get_lut(lut_path(lut), "cuda").handle, x.data_ptr(), dy.data_ptr(),
                                                   dw.data_ptr(), rows, units, width, ws.data_ptr(), ws.numel(), 0))
        return dw
    assert torch.equal(grad(0), grad(128 << 20))


def test_every_shipped_table_takes_the_path(forced):
    """With AMSIM_CODES=0 the table kernels run: another order of the same sum, so the bits differ."""
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.randn(256, 300, generator=g, device="cuda"), torch.randn(300, 256, generator=g, device="cuda")
    for lut in ("ACC_7", "MBM_3", "MBM_5", "MBM_7", "MIT_3", "MIT_5", "MIT_7"):
        os.environ["AMSIM_CODES"] = "1"
        forced.lib.amsim_debug_reload_env()
        a = ops.denseam(x, w, lut_path(lut))
        os.environ["AMSIM_CODES"] = "0"
        forced.lib.amsim_debug_reload_env()
        b = ops.denseam(x, w, lut_path(lut))
        assert not torch.equal(a, b), lut
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-5
    assert np.isfinite(a.cpu().numpy()).all()


def test_a_wait_that_runs_out_is_reported_by_the_next_call(forced, monkeypatch):
    """With no tries at all every warp gives up at its first wait: the launch ends, and the next call says so, once."""
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w, lut = torch.randn(600, 300, generator=g, device="cuda"), torch.randn(300, 200, generator=g, device="cuda"), lut_path("MBM_7")
    want = ops.denseam(x, w, lut)
    monkeypatch.setenv("AMSIM_CODES_SPIN", "0")
    forced.lib.amsim_debug_reload_env()
    ops.denseam(x, w, lut)
    torch.cuda.synchronize()
    monkeypatch.delenv("AMSIM_CODES_SPIN")
    forced.lib.amsim_debug_reload_env()
    with pytest.raises(ops.AmsimError, match="gave up waiting"):
        ops.denseam(x, w, lut)
    assert torch.equal(ops.denseam(x, w, lut), want)      # (the tile counters are in step)
    assert forced.lib.amsim_async_status() == 0


def _products(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [(torch.randn(1200 + 100 * i, 700, generator=g, device="cuda"), torch.randn(700, 300, generator=g, device="cuda"))
            for i in range(n)]


@pytest.mark.parametrize("codes", [1, 0])
def test_captured_launches_on_forked_branches_do_not_share_scratch(forced, codes):
    """Tiles of one branch parked among the other's would show as wrong sums; eager launches have scratch of their own."""
    from approxtrain_b200 import ops
    lut = lut_path("MBM_7")
    _on(forced, codes, lambda: None)
    pairs = _products(4, 1)
    want = [ops.denseam(x, w, lut) for x, w in pairs]
    torch.cuda.synchronize()
    graph, out = torch.cuda.CUDAGraph(), [None] * len(pairs)
    side = [torch.cuda.Stream() for _ in pairs[1:]]
    with torch.cuda.graph(graph):
        here = torch.cuda.current_stream()
        for i, s in enumerate(side):
            s.wait_stream(here)
            with torch.cuda.stream(s):
                out[i + 1] = ops.denseam(*pairs[i + 1], lut)
                out[i + 1] = ops.denseam(*pairs[i + 1], lut)     # (a second launch of the stream takes the same region)
        out[0] = ops.denseam(*pairs[0], lut)
        for s in side:
            here.wait_stream(s)
    for _ in range(20):
        for o in out:
            o.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want))


def test_graphs_replayed_side_by_side_do_not_share_scratch_and_give_it_back(forced):
    from approxtrain_b200 import ops
    lut = lut_path("MIT_7")
    pairs = _products(2, 2)
    want = [ops.denseam(x, w, lut) for x, w in pairs]
    free = []
    for round_ in range(8):
        graphs, outs = [], []
        for x, w in pairs:
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1]):
                outs.append(ops.denseam(x, w, lut))
        streams = [torch.cuda.Stream() for _ in pairs]
        for _ in range(10):
            for s, gr in zip(streams, graphs):
                s.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(s):
                    gr.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(outs, want))
        del graphs, outs, gr
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free.append(torch.cuda.mem_get_info()[0])
    assert min(free[2:]) >= free[1] - (4 << 20), free      # later captures use what earlier graphs gave back


SOME = [(2, 9, 13, 16, 3, 3, 65, 1, "SAME"), (1, 30, 30, 3, 7, 7, 64, 2, "VALID"), (3, 11, 7, 8, 3, 3, 129, 2, "SAME"), (2, 14, 14, 64, 1, 1, 300, 1, "VALID")]


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7"])
@pytest.mark.parametrize("shape", SOME)
def test_fused_epilogue_equals_the_separate_operations(forced, lut, shape):
    from approxtrain_b200 import ops
    n, h, w, c, kh, kw, k, s, pad = shape
    g = torch.Generator(device="cuda").manual_seed(k)
    x, wt = torch.randn(n, h, w, c, generator=g, device="cuda"), torch.randn(kh, kw, c, k, generator=g, device="cuda")
    b, sc = torch.randn(k, generator=g, device="cuda"), torch.rand(k, generator=g, device="cuda") - 0.3
    kw_ = dict(strides=s, padding=pad, mant_mul_lut=lut_path(lut))
    y = ops.convam(x, wt, **kw_)
    assert torch.equal(ops.convam_bias_act(x, wt, b, activation="relu", scale=sc, **kw_), torch.relu(y * sc + b))
    assert torch.equal(ops.convam_bias_act(x, wt, b, **kw_), y + b)
    if kh == 1:
        flat, mat = x.reshape(-1, c), wt[0, 0]
        assert torch.equal(ops.denseam_bias_act(flat, mat, b, activation="relu", mant_mul_lut=lut_path(lut)),
                           torch.relu(ops.denseam(flat, mat, lut_path(lut)) + b))


def _off_by_one_float(t):
    room = torch.empty(t.numel() + 1, device="cuda")
    view = room[1:].view(t.shape)
    view.copy_(t)
    assert view.data_ptr() % 16 == 4
    return view


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_5"])
@pytest.mark.parametrize("shape", SOME)
def test_operands_off_16_byte_alignment(forced, lut, shape):
    """Element-wise fetches of what aligned operands fetch 16 bytes at a time: the same sums in the same order."""
    from approxtrain_b200 import ops
    n, h, w, c, kh, kw, k, s, pad = shape
    g = torch.Generator(device="cuda").manual_seed(c)
    x, wt = torch.randn(n, h, w, c, generator=g, device="cuda"), torch.randn(kh, kw, c, k, generator=g, device="cuda")
    kw_ = dict(strides=s, padding=pad, mant_mul_lut=lut_path(lut))
    y = ops.convam(x, wt, **kw_)
    dy = torch.randn(y.shape, generator=g, device="cuda")
    dx, dw = ops.convam_input_grad(x.shape, wt, dy, **kw_), ops.convam_filter_grad(wt.shape, x, dy, **kw_)
    for f in (lambda t: t, _off_by_one_float):
        for e in (lambda t: t, _off_by_one_float):
            assert torch.equal(ops.convam(f(x), e(wt), **kw_), y)
            assert torch.equal(ops.convam_input_grad(x.shape, e(wt), f(dy), **kw_), dx)
            assert torch.equal(ops.convam_filter_grad(wt.shape, f(x), e(dy), **kw_), dw)


@pytest.mark.parametrize("lut", ["MBM_7", "MIT_7", "MBM_5"])
@pytest.mark.parametrize("rows,width,units", [(300, 64, 257), (257, 500, 64), (130, 33, 300), (1000, 129, 130)])
def test_dense_gradients_in_either_operand_role(forced, lut, rows, width, units):
    from approxtrain_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, w = torch.randn(rows, width, generator=g, device="cuda"), torch.randn(width, units, generator=g, device="cuda")
    dy = torch.randn(rows, units, generator=g, device="cuda")
    for got, want in zip(ops.denseam_grad(dy, x, w, lut_path(lut)), ops.denseam_grad(dy, x, w, lut_path(lut), deterministic=True)):
        _close(got, want)


def test_offsets_beyond_31_bits(forced):
    from approxtrain_b200 import ops
    rows = (1 << 31) // 64 + 5000
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB")
    g = torch.Generator(device="cuda").manual_seed(5)
    w = torch.randn(64, 64, generator=g, device="cuda")
    x = torch.randn(rows, 64, generator=g, device="cuda")
    y = ops.denseam(x, w, lut_path("MBM_7"))
    for part in (slice(0, 3000), slice(rows // 2, rows // 2 + 3000), slice(rows - 3000, rows)):
        _close(y[part], ops.denseam(x[part], w, lut_path("MBM_7"), deterministic=True))
    dw = ops.denseam_grad(y, x, w, lut_path("MBM_7"))[1]        # the reduction runs over all rows
    want = sum(ops.denseam_grad(y[i:i + rows // 4 + 1], x[i:i + rows // 4 + 1], w, lut_path("MBM_7"))[1].double()
               for i in range(0, rows, rows // 4 + 1))
    _close(dw, want)
