"""FrozenMatmul on the GPU (through the C ABI) against the CPU oracle.

Mirrors the reference's own checks: backward_input equals the dense dy.W built from row()
(tests/engine.rs:96-120, tolerance 1e-3), the adjoint identity (src/frozen.rs:218-227), and
shape refusals (the reference panics; here a status).  Rows are bit exact (byte/integer
work); matmuls use f16 operands with f32 accumulation, tolerance 2e-3 relative L2.
"""
import numpy as np
import pytest

import rust_trainer_b200 as rt
from conftest import rel_l2
from oracle import oracle as O
from rust_trainer_b200 import quants as Q

pytestmark = pytest.mark.gpu

FORMATS = [Q.F16, Q.BF16, Q.Q8_0, Q.Q4_0, Q.Q4_K, Q.Q6_K]
MATMUL_TOL = 2e-3


def _shapes(t):
    pair = [(1024, 512, 2500), (512, 512, 5001)]  # enough 256-row tiles for the CTA-pair kernel
    if t in (Q.Q4_K, Q.Q6_K):
        return [(128, 256, 40), (384, 512, 300), (1024, 1024, 513)] + pair
    return [(128, 64, 1), (256, 128, 100), (192, 96, 7), (896, 896, 300), (1024, 1024, 513)] + pair


@pytest.mark.parametrize("t", FORMATS, ids=[Q.NAMES[t] for t in FORMATS])
def test_rows_are_bit_exact(ctx, t):
    rng = np.random.default_rng(t)
    n, k = 200, 512
    packed = Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t)
    want = O.dequant_rows(t, packed, n, k)
    f = rt.Frozen(ctx, t, n, k, packed)
    assert (f.out_dim(), f.in_dim(), f.nbytes()) == (n, k, packed.size)
    for r in (0, 1, 63, 64, 127, 128, 199):
        assert np.array_equal(f.row(r), want[r]), r
    with pytest.raises(rt.RtError) as e:
        f.row(n)
    assert e.value.status == 6
    f.close()


@pytest.mark.parametrize("t", FORMATS, ids=[Q.NAMES[t] for t in FORMATS])
def test_forward_and_backward_input(ctx, t):
    rng = np.random.default_rng(100 + t)
    for n, k, m in _shapes(t):
        packed = Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t)
        f = rt.Frozen(ctx, t, n, k, packed)
        x = rng.standard_normal((m, k)).astype(np.float32)
        assert rel_l2(f.forward(x, m), O.frozen_forward(t, n, k, packed, x, m)) < MATMUL_TOL, (n, k, m)
        dy = rng.standard_normal((m, n)).astype(np.float32)
        dx0 = rng.standard_normal((m, k)).astype(np.float32)
        dx, ref = dx0.copy(), dx0.copy()
        f.backward_input(dy, m, dx)  # accumulates, like the trait method
        O.frozen_backward_input(t, n, k, packed, dy, m, ref)
        assert rel_l2(dx, ref) < MATMUL_TOL, (n, k, m)
        f.close()


@pytest.mark.parametrize("t", [Q.Q8_0, Q.Q4_0, Q.Q6_K])
def test_adjoint_identity_on_device(ctx, t):
    rng = np.random.default_rng(7)
    n, k, m = 384, 512, 33
    f = rt.Frozen.from_f32(ctx, (rng.standard_normal((n, k)) * 0.1).astype(np.float32), t)
    x = rng.standard_normal((m, k)).astype(np.float32)
    dy = rng.standard_normal((m, n)).astype(np.float32)
    y = f.forward(x, m)
    dx = np.zeros((m, k), np.float32)
    f.backward_input(dy, m, dx)
    lhs, rhs = float((dy.astype(np.float64) * y).sum()), float((dx.astype(np.float64) * x).sum())
    assert abs(lhs - rhs) <= 2e-3 * max(1.0, abs(lhs))
    f.close()


@pytest.mark.parametrize("n,k,tokens", [(512, 256, 300), (384, 256, 1000), (1024, 128, 4133), (1024, 512, 4133)])
def test_16_bit_outputs_are_the_rounded_f32_outputs(ctx, n, k, tokens):
    """The device entry points write f32, f16 or bf16.  The 16-bit epilogue (fragment-layout TMEM
    loads, paired rounding, transposing matrix stores, swizzled TMA store) must give exactly the
    f32 result rounded once, for the CTA-pair kernel (a multiple of 256 features), the single-CTA
    one, and token counts that end inside a tile and inside a 32-token block."""
    import torch

    from rust_trainer_b200._lib import DT_BF16, DT_F16, DT_F32, lib

    L = lib()
    rng = np.random.default_rng(n + tokens)
    f = rt.Frozen.from_f32(ctx, (rng.standard_normal((n, k)) * 0.05).astype(np.float32), Q.Q8_0)
    x = torch.randn(tokens, k, device="cuda", dtype=torch.float16)
    y32 = torch.full((tokens, n), float("nan"), device="cuda", dtype=torch.float32)
    torch.cuda.synchronize()
    ctx.check(L.rt_frozen_forward_dev(f._h, x.data_ptr(), DT_F16, tokens, y32.data_ptr(), DT_F32, 0))
    for dt, tdt in ((DT_F16, torch.float16), (DT_BF16, torch.bfloat16)):
        assert (f.tile(tokens, False, DT_F16, dt)[0] == "pair") == (k == 512)
        y16 = torch.full((tokens + 1, n), 7.0, device="cuda", dtype=tdt)  # one guard row behind the output
        torch.cuda.synchronize()
        ctx.check(L.rt_frozen_forward_dev(f._h, x.data_ptr(), DT_F16, tokens, y16.data_ptr(), dt, 0))
        ctx.synchronize()
        assert torch.equal(y16[:tokens], y32.to(tdt)), (dt, float((y16[:tokens].float() - y32).abs().max()))
        assert bool((y16[tokens] == 7.0).all())  # nothing written past the last token
    f.close()


def test_empty_and_refused_inputs(ctx):
    rng = np.random.default_rng(0)
    w = (rng.standard_normal((64, 64)) * 0.02).astype(np.float32)
    f = rt.Frozen.from_f32(ctx, w, Q.Q4_0)
    assert f.forward(np.zeros((0, 64), np.float32), 0).shape == (0, 64)  # t = 0 is a no-op
    with pytest.raises(rt.RtError):
        f.forward(np.zeros((3, 32), np.float32), 3)  # wrong inner dimension
    f.close()
    packed = Q.quantize(w, Q.Q4_0)
    with pytest.raises(rt.RtError) as e:
        rt.Frozen(ctx, 3, 64, 64, packed)  # Q4_1: unsupported
    assert e.value.status == 2
    with pytest.raises(rt.RtError) as e:
        rt.Frozen(ctx, Q.Q4_0, 64, 64, packed[:-1])  # byte count does not match
    assert e.value.status == 1
    with pytest.raises(rt.RtError) as e:
        rt.Frozen(ctx, Q.Q4_K, 4, 128, np.zeros(4 * 72, np.uint8))  # 128 is not a multiple of 256
    assert e.value.status == 1


def test_full_size_properties(ctx):
    """The benchmark's sizes (ffn_gate of the 0.6B shape, 3072 x 1024, at 8192 tokens), checked by
    properties that do not need the oracle: linearity in x and the adjoint identity."""
    rng = np.random.default_rng(3)
    n, k, m = 3072, 1024, 8192
    f = rt.Frozen.from_f32(ctx, (rng.standard_normal((n, k)) * 0.02).astype(np.float32), Q.Q8_0)
    x1 = rng.standard_normal((m, k)).astype(np.float32)
    x2 = rng.standard_normal((m, k)).astype(np.float32)
    y1, y2, y12 = f.forward(x1, m), f.forward(x2, m), f.forward(x1 + x2, m)
    assert rel_l2(y12, y1 + y2) < MATMUL_TOL
    dy = rng.standard_normal((m, n)).astype(np.float32)
    dx = np.zeros((m, k), np.float32)
    f.backward_input(dy, m, dx)
    lhs, rhs = float((dy.astype(np.float64) * y1).sum()), float((dx.astype(np.float64) * x1).sum())
    assert abs(lhs - rhs) <= 2e-3 * abs(lhs) + 50.0  # inner products of ~2.5e7 random terms
    f.close()


def test_a_wait_that_runs_out_is_a_status_not_a_hang(ctx):
    """Every device-side wait is bounded: a barrier nothing arrives on makes the wait give up after
    its limit (here 2e8 cycles, about 0.1 s), the kernel returns, the host reads
    RT_ERR_DEVICE_WAIT_TIMEOUT with the wait's site code, and the context keeps working."""
    from rust_trainer_b200._lib import lib

    st = lib().rt_ctx_selftest_wait_timeout(ctx._h, 200_000_000)
    assert st == 5  # RT_ERR_DEVICE_WAIT_TIMEOUT
    assert b"site 999" in lib().rt_last_error(ctx._h)
    rng = np.random.default_rng(1)
    w = (rng.standard_normal((128, 64)) * 0.02).astype(np.float32)
    f = rt.Frozen.from_f32(ctx, w, Q.Q8_0)
    x = rng.standard_normal((5, 64)).astype(np.float32)
    assert rel_l2(f.forward(x, 5), x @ O.dequant_rows(Q.Q8_0, Q.quantize(w, Q.Q8_0), 128, 64).T) < MATMUL_TOL
    f.close()


def test_builtin_f32_and_q8_0_weights(ctx):
    """FrozenWeight::{F32, Q8_0} (src/frozen.rs:33-187) with the reference's own unit test
    (src/frozen.rs:206-228): Q8_0 forward within 0.02 of f32, and the adjoint identity
    <dy, x.W^T> == <dy.W, x> to 1e-3 for both storages; plus exact rows and the oracle."""
    r = O.Rng(3)
    out, inp, t = 8, 64, 3  # the reference's test has 6 rows; 16-bit operand rows must be a multiple of 8 long here
    w = r.vec_normal(out * inp, 0.1).reshape(out, inp)
    x = r.vec_normal(t * inp, 1.0).reshape(t, inp)
    dy = r.vec_normal(t * out, 1.0).reshape(t, out)
    f = rt.Frozen.f32(ctx, w)
    q = rt.Frozen.q8_0(ctx, w)
    assert f.nbytes() == out * inp * 4 and q.nbytes() == out * inp // 32 * 4 + out * inp  # src/frozen.rs:181-186
    yf, yq = f.forward(x, t), q.forward(x, t)
    assert np.max(np.abs(yf - yq)) < 0.02
    assert rel_l2(yf, x @ w.T) < 1e-3
    for wq in (f, q):
        y = wq.forward(x, t)
        dx = np.zeros((t, inp), np.float32)
        wq.backward_input(dy, t, dx)
        lhs, rhs = float((dy * y).sum()), float((dx * x).sum())
        assert abs(lhs - rhs) < 1e-3 * max(abs(lhs), 1.0)
    assert np.array_equal(f.row(4), w[4])
    from rust_trainer_b200.frozen import quantize_q8_0_f32scale

    d, qs = quantize_q8_0_f32scale(w)
    deq = (np.repeat(d, 32) * qs.astype(np.float32)).reshape(out, inp)
    assert np.array_equal(q.row(5), deq[5])
    f.close()
    q.close()
    # a wide f32 weight against the oracle's F32 rows, both directions
    rng = np.random.default_rng(9)
    n, k, m = 384, 1024, 300
    w2 = (rng.standard_normal((n, k)) * 0.05).astype(np.float32)
    x2 = rng.standard_normal((m, k)).astype(np.float32)
    dy2 = rng.standard_normal((m, n)).astype(np.float32)
    f2 = rt.Frozen.f32(ctx, w2)
    assert rel_l2(f2.forward(x2, m), O.frozen_forward(0, n, k, w2, x2, m)) < MATMUL_TOL
    dx, ref = np.zeros((m, k), np.float32), np.zeros((m, k), np.float32)
    f2.backward_input(dy2, m, dx)
    O.frozen_backward_input(0, n, k, w2, dy2, m, ref)
    assert rel_l2(dx, ref) < MATMUL_TOL
    f2.close()


@pytest.mark.parametrize("t,n,k,big", [(Q.Q4_0, 320, 704, 2600), (Q.Q8_0, 320, 704, 2600), (Q.Q4_K, 192, 768, 2600), (Q.Q6_K, 1088, 768, 1300),
                                       (Q.F16, 320, 704, 2600), (Q.BF16, 320, 704, 2600), (Q.F16, 128, 64, 40000), (Q.Q4_0, 1088, 704, 2600),
                                       (Q.Q8_0, 1088, 704, 2600), (Q.Q4_K, 1088, 768, 2600), (Q.Q6_K, 1088, 768, 2600), (Q.F16, 1088, 704, 2600)],
                         ids=lambda v: Q.NAMES.get(v, v) if isinstance(v, int) and v < 64 else str(v))
def test_a_row_gets_the_same_bits_in_any_batch(ctx, t, n, k, big):
    """An output element is one accumulation chain whatever tile it falls into, so every tile kind, unpacking into shared memory
    or into TMEM, has to give the same bits: batches of sizes around the tile edges (32 and 64 tokens; half, narrow and pair
    tiles; an odd number of 64-element steps; rows that end inside a tile; several tiles per CTA) against one large batch."""
    rng = np.random.default_rng(n + k)
    packed = Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t)
    f = rt.Frozen(ctx, t, n, k, packed)
    x = rng.standard_normal((big, k)).astype(np.float32)
    dy = rng.standard_normal((big, n)).astype(np.float32)
    y = f.forward(x, big)
    dx = np.zeros((big, k), np.float32)
    f.backward_input(dy, big, dx)
    rows = rng.integers(0, big, 64)
    assert rel_l2(y[rows], O.frozen_forward(t, n, k, packed, x[rows], 64)) < MATMUL_TOL
    sizes = (1, 31, 33, 64, 65, 157, 640, 1100)
    if (n, big) == (1088, 2600):
        kinds = {f.tile(m, backward)[0] for m in sizes + (big,) for backward in (False, True)}
        assert f.tile(big)[0] == f.tile(big, True)[0] == "pair" and ({"half", "narrow"} if t == Q.F16 else {"half", "slim", "narrow_tmem"}) <= kinds, kinds
    for m in sizes:
        at = big - m
        assert np.array_equal(f.forward(x[at:], m), y[at:]), m
        part = np.zeros((m, k), np.float32)
        f.backward_input(dy[at:], m, part)
        assert np.array_equal(part, dx[at:]), m
    f.close()


SLIM_ROWS = (1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 250)
SLIM = [(t, 712, 6400, False, SLIM_ROWS) for t in (Q.Q4_0, Q.Q4_K, Q.Q6_K, Q.F16)]
SLIM += [(Q.Q4_0, 6400, 672, True, SLIM_ROWS), (Q.Q4_K, 6400, 768, True, SLIM_ROWS), (Q.Q6_K, 6400, 768, True, SLIM_ROWS), (Q.F16, 6400, 712, True, SLIM_ROWS)]
SLIM += [(Q.Q8_0, 1088, 704, True, (1055, 1089, 1100))]


@pytest.mark.parametrize("t,n,k,backward,rows", SLIM, ids=[f"{Q.NAMES[c[0]]}-{c[1]}x{c[2]}" for c in SLIM])
def test_slim_pair_tiles_at_their_edges(ctx, t, n, k, backward, rows):
    """Tiles of 128 weight rows over a CTA pair whose accumulator holds the two halves of the tokens in the two halves of its
    lanes: tokens that end inside a tile, at its half and inside a block, rows that end inside a tile and inside a CTA's half;
    f32, 16-bit (by TMA, and at an address it does not take) and accumulated results have the bits of 256-row pair tiles."""
    import torch

    from rust_trainer_b200._lib import DT_BF16, DT_F16, DT_F32, lib

    L, big = lib(), 2600
    g = torch.Generator(device="cuda").manual_seed(n + k)
    packed = Q.quantize((np.random.default_rng(n + k).standard_normal((n, k)) * 0.05).astype(np.float32), t)
    f = rt.Frozen(ctx, t, n, k, packed)
    call = L.rt_frozen_backward_input_dev if backward else L.rt_frozen_forward_dev
    ci, co = (n, k) if backward else (k, n)
    x, want = torch.randn(big, ci, generator=g, device="cuda").half(), torch.empty(big, co, device="cuda")
    torch.cuda.synchronize()
    ctx.check(call(f._h, x.data_ptr(), DT_F16, big, want.data_ptr(), DT_F32, 0))
    ctx.synchronize()
    assert f.tile(big, backward)[0] == "pair"
    w = torch.from_numpy(O.dequant_rows(t, packed, n, k)).cuda().double()
    assert rel_l2(want[-250:].cpu().numpy(), (x[-250:].double() @ (w if backward else w.T)).cpu().numpy()) < MATMUL_TOL
    widths = set()
    for m in rows:
        part, exp = x[big - m:], want[big - m:]

        def run(out_dtype, out, accumulate=0):
            kind, width = f.tile(m, backward, DT_F16, out_dtype)
            assert kind == "slim", (m, kind)
            widths.add(width)
            torch.cuda.synchronize()
            ctx.check(call(f._h, part.data_ptr(), DT_F16, m, out.data_ptr(), out_dtype, accumulate))
            ctx.synchronize()

        for dt, tdt in ((DT_F32, torch.float32), (DT_F16, torch.float16), (DT_BF16, torch.bfloat16)):
            y = torch.full((m + 1, co), 7.0, device="cuda", dtype=tdt)  # one guard row behind the results
            run(dt, y)
            assert torch.equal(y[:m], exp.to(tdt)) and bool((y[m] == 7.0).all()), (m, dt)
        odd = torch.full(((m + 1) * co + 1,), 7.0, device="cuda", dtype=torch.float16)[1:].view(m + 1, co)
        run(DT_F16, odd)
        assert torch.equal(odd[:m], exp.half()) and bool((odd[m] == 7.0).all()), m
        base = torch.randn(m + 1, co, generator=g, device="cuda")
        acc = base.clone()
        run(DT_F32, acc, 1)
        assert torch.equal(acc[:m], base[:m] + exp) and torch.equal(acc[m], base[m]), m
    if rows is SLIM_ROWS:
        assert widths == {32, 64, 128}
    f.close()


# products whose other kinds of tile took at least 5 % longer, behind themselves and behind a kernel that lets nothing start under it
MEASURED = [(Q.Q4_0, 3072, 1024, False, 400, "pair"), (Q.Q4_K, 2048, 1024, False, 700, "pair"), (Q.Q6_K, 4096, 1024, False, 400, "pair slim"),
            (Q.Q4_0, 1024, 1024, False, 2048, "pair slim"), (Q.Q6_K, 1024, 3072, False, 1024, "slim"), (Q.Q6_K, 2048, 1024, True, 1024, "slim"),
            (Q.F16, 4864, 896, True, 64, "slim"), (Q.F16, 1024, 3072, False, 64, "slim"), (Q.Q8_0, 6144, 1024, True, 8, "half"),
            (Q.Q8_0, 8192, 3072, True, 24, "half")]


@pytest.mark.parametrize("t,n,k,backward,m,kinds", MEASURED, ids=lambda v: str(v))
def test_tile_choice_is_a_kind_that_measured_fastest(ctx, t, n, k, backward, m, kinds):
    f = rt.Frozen(ctx, t, n, k, np.zeros(rt.lib().rt_ggml_nbytes(t, n, k), np.uint8))
    assert f.tile(m, backward)[0] in kinds.split()
    f.close()


def test_results_in_locked_memory_are_the_callers(ctx):
    """Results of 64 KB and more lie in page-locked blocks of a bounded pool: a block is reused only after the last view of it
    is gone, and past the bound (256 MB) results come in ordinary memory."""
    rng = np.random.default_rng(0)
    n, k, m = 4096, 64, 2048  # 32 MB of results
    f = rt.Frozen.from_f32(ctx, (rng.standard_normal((n, k)) * 0.02).astype(np.float32), Q.Q8_0)
    xs = [rng.standard_normal((m, k)).astype(np.float32) for _ in range(10)]
    ys = [f.forward(x, m) for x in xs]  # 320 MB held at once
    for x, y in zip(xs, ys):
        assert np.array_equal(f.forward(x, m), y)
    view = ys[0][5:7]
    keep = view.copy()
    del y, ys
    for x in xs:
        f.forward(x, m)
    assert np.array_equal(view, keep)
    f.close()


OUTLIVES = """
import ctypes as C
import numpy as np
import rust_trainer_b200 as rt
from rust_trainer_b200 import quants as Q
cudart = C.CDLL("libcudart.so.12")
def locked(address):
    attr = (C.c_uint64 * 16)()  # cudaPointerAttributes: the memory's type comes first, 0 for ordinary memory
    assert cudart.cudaPointerGetAttributes(attr, C.c_void_p(address)) == 0
    return C.cast(attr, C.POINTER(C.c_int))[0] != 0
ctx = rt.Context(0)
f = rt.Frozen.from_f32(ctx, np.ones((1024, 64), np.float32), Q.Q8_0)
y, z = (f.forward(np.ones((m, 64), np.float32), m) for m in (64, 128))
at_y, at_z = y.ctypes.data, z.ctypes.data
assert locked(at_y) and locked(at_z)
del z
assert locked(at_z)  # waits in the pool for the next result
f.close()
ctx.close()
assert not locked(at_z) and locked(at_y) and float(y[3, 5]) == float(y[0, 0])
del y
assert not locked(at_y)
"""


def test_a_result_that_outlives_its_context_is_unlocked_with_its_last_view():
    import subprocess
    import sys

    subprocess.run([sys.executable, "-c", OUTLIVES], check=True, timeout=300)


@pytest.mark.parametrize("nbytes", [(256 << 20) + 1, 1 << 60, (1 << 64) - 1])
def test_locked_memory_past_the_pools_bound_is_refused(ctx, nbytes):
    assert not rt.lib().rt_host_alloc(ctx._h, nbytes)
    block = rt.lib().rt_host_alloc(ctx._h, 65536)
    assert block
    rt.lib().rt_host_free(block)
