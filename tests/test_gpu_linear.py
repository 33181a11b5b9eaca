"""Linear + LoRA on the GPU against the oracle's restatement of src/linear.rs:73-121.

Tolerances: outputs and dx 2e-3 relative L2 (f16 operands, f32 accumulation); adapter
gradients 5e-3 relative L2 and cosine >= 0.9999 (the north-star bar is 1e-2 / 0.999).
"""
import numpy as np
import pytest

import rust_trainer_b200 as rt
from conftest import cosine, rel_l2
from oracle import oracle as O
from rust_trainer_b200 import quants as Q

pytestmark = pytest.mark.gpu

CASES = [(Q.Q4_0, 256, 128, 50, 8), (Q.Q8_0, 3072, 1024, 700, 16), (Q.Q6_K, 512, 1024, 300, 32),
         (Q.F16, 384, 256, 100, 16), (Q.BF16, 256, 256, 65, 4), (Q.Q4_K, 1024, 768, 257, 16), (Q.Q8_0, 128, 896, 1, 64),
         # enough 256-row tiles for the CTA-pair kernel, ragged token counts, packed and 16-bit weights
         (Q.Q8_0, 1024, 512, 2500, 16), (Q.Q4_0, 512, 512, 5001, 8), (Q.F16, 768, 512, 3300, 16),
         (Q.Q6_K, 512, 1024, 4999, 32), (Q.Q4_K, 1280, 256, 2047, 64)]


def _make(ctx, rng, t, n, k, r, bias=True):
    packed = Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t)
    b = (rng.standard_normal(n) * 0.01).astype(np.float32) if bias else None
    a_ = (rng.standard_normal((r, k)) / r).astype(np.float32)
    b_ = (rng.standard_normal((n, r)) * 0.05).astype(np.float32)
    f = rt.Frozen(ctx, t, n, k, packed)
    lin = rt.Linear("blk.0.test", f, b)
    lin.attach_lora(r, 2.0 * r, a_, b_)
    return packed, b, a_, b_, f, lin


@pytest.mark.parametrize("t,n,k,m,r", CASES, ids=[f"{Q.NAMES[c[0]]}-{c[1]}x{c[2]}-t{c[3]}-r{c[4]}" for c in CASES])
def test_forward_backward_with_adapter(ctx, t, n, k, m, r):
    rng = np.random.default_rng(n + k + m + r)
    packed, bias, a, b, f, lin = _make(ctx, rng, t, n, k, r)
    alpha = 2.0 * r
    x = rng.standard_normal((m, k)).astype(np.float32)
    assert rel_l2(lin.forward(x, m), O.linear_forward(t, n, k, packed, bias, r, alpha, a, b, x, m)) < 2e-3
    # gradients spanning five orders of magnitude between rows: the per-row scaling must hold
    dy = (rng.standard_normal((m, n)) * 1e-3 * np.exp(rng.standard_normal((m, 1)) * 2.5)).astype(np.float32)
    dx = lin.backward(x, dy, m)
    ga, gb = np.zeros_like(a), np.zeros_like(b)
    dxo = O.linear_backward(t, n, k, packed, r, alpha, a, b, ga, gb, x, dy, m)
    got = lin.lora()
    assert rel_l2(dx, dxo) < 2e-3
    assert rel_l2(got["ga"], ga) < 5e-3 and cosine(got["ga"], ga) > 0.9999
    assert rel_l2(got["gb"], gb) < 5e-3 and cosine(got["gb"], gb) > 0.9999
    # a second backward accumulates into ga / gb (src/linear.rs:108,113)
    lin.backward(x, dy, m)
    got2 = lin.lora()
    assert rel_l2(got2["ga"], 2 * ga) < 5e-3 and rel_l2(got2["gb"], 2 * gb) < 5e-3
    lin.zero_grad()
    z = lin.lora()
    assert not z["ga"].any() and not z["gb"].any()
    lin.close()
    f.close()


def test_adapter_bypass_and_fresh_adapter_is_a_no_op(ctx):
    rng = np.random.default_rng(5)
    t, n, k, m, r = Q.Q8_0, 256, 256, 40, 8
    packed, bias, a, b, f, lin = _make(ctx, rng, t, n, k, r)
    x = rng.standard_normal((m, k)).astype(np.float32)
    base = O.linear_forward(t, n, k, packed, bias, 0, 1.0, None, None, x, m)
    lin.set_lora_enabled(False)  # src/linear.rs:64-70
    assert rel_l2(lin.forward(x, m), base) < 2e-3
    dy = rng.standard_normal((m, n)).astype(np.float32)
    lin.backward(x, dy, m)
    g = lin.lora()
    assert not g["ga"].any() and not g["gb"].any()  # no gradient while bypassed
    lin.set_lora_enabled(True)
    lin.write_lora(None, np.zeros_like(b))  # B = 0: PEFT-style init, exact no-op on the output
    assert rel_l2(lin.forward(x, m), base) < 2e-3
    lin.close()
    f.close()


def test_shape_errors_are_statuses(ctx):
    rng = np.random.default_rng(6)
    f = rt.Frozen.from_f32(ctx, (rng.standard_normal((64, 64)) * 0.02).astype(np.float32), Q.Q4_0)
    with pytest.raises(rt.RtError):
        rt.Linear("bad", f, np.zeros(3, np.float32))  # src/linear.rs:49-51 asserts bias length
    lin = rt.Linear("ok", f)
    with pytest.raises(rt.RtError):
        lin.attach_lora(8, 16.0, np.zeros((8, 32), np.float32), np.zeros((64, 8), np.float32))
    with pytest.raises(rt.RtError) as e:
        lin.attach_lora(65, 16.0, np.zeros((65, 64), np.float32), np.zeros((64, 65), np.float32))
    assert e.value.status == 7
    with pytest.raises(rt.RtError):
        lin.forward(np.zeros((2, 63), np.float32), 2)
    lin.close()
    f.close()


@pytest.mark.parametrize("t,n,k,m,r", [(Q.Q8_0, 128, 256, 9000, 16), (Q.Q8_0, 128, 3072, 4200, 40), (Q.Q4_0, 192, 512, 2049, 3),
                                       (Q.F16, 264, 72, 65, 64), (Q.Q4_0, 128, 64, 1025, 16)])
def test_adapter_streams_at_the_edges_of_their_splits(ctx, t, n, k, m, r):
    """Low-rank streams and adapter gradients where their split changes: more than eight 1024-token splits, one token past a
    split and past the 2048 and 4096 tokens at which the streams' tiles grow, contraction pieces of a wide input, ranks that
    are no multiple of 16, column tiles that end inside a matrix."""
    test_forward_backward_with_adapter(ctx, t, n, k, m, r)


@pytest.mark.parametrize("t,n,k,m,r", [(Q.Q8_0, 256, 512, 300, 16), (Q.F16, 384, 256, 2500, 8)])
def test_dx_may_be_written_over_x(ctx, t, n, k, m, r):
    """On device buffers dx may take the memory of an x that is needed no more: the adapter gradients are those of separate buffers."""
    import torch

    rng = np.random.default_rng(9)
    _, _, _, _, f, lin = _make(ctx, rng, t, n, k, r)
    x = torch.randn(m, k, generator=torch.Generator().manual_seed(1)).half().cuda()
    dy = torch.randn(m, n, generator=torch.Generator().manual_seed(2)).half().cuda()

    def run(x16, dx):
        lin.zero_grad()
        torch.cuda.synchronize()
        ctx.check(rt.lib().rt_linear_backward_dev(lin._h, x16.data_ptr(), dy.data_ptr(), None, m, dx.data_ptr(), 0))
        ctx.synchronize()
        got = lin.lora()
        return dx.clone(), got["ga"].copy(), got["gb"].copy()

    want = run(x, torch.empty(m, k, device="cuda"))
    for at in (0, m * k // 8 * 8):  # the first or the second half of the result's memory
        both = torch.empty(m * k, device="cuda")
        x16 = both.view(torch.float16)[at:at + m * k].view(m, k)
        x16.copy_(x)
        got = run(x16, both.view(m, k))
        assert torch.equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    lin.close()
    f.close()


def test_a_contexts_scratch_goes_with_it():
    """What linears outside a model work in belongs to their context: it is freed with it, and a later context, which may get the
    same address and another device, does not find it."""
    import torch

    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def use():
        c = rt.Context(0)
        f = rt.Frozen.from_f32(c, np.ones((64, 64), np.float32), Q.Q8_0)
        lin = rt.Linear("l", f)
        lin.attach_lora(8, 16.0, np.zeros((8, 64), np.float32), np.zeros((64, 8), np.float32))
        x = torch.zeros(1 << 20, 64, dtype=torch.float16, device="cuda")
        y = torch.empty(1 << 20, 64, dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        c.check(rt.lib().rt_linear_forward_dev(lin._h, x.data_ptr(), 1 << 20, y.data_ptr(), 2, 0))  # 192 MB of Hs
        c.synchronize()
        lin.close()
        f.close()
        held = free_bytes()
        c.close()
        return held

    use()
    before = free_bytes()
    assert use() < before - (100 << 20)
    assert abs(free_bytes() - before) < 32 << 20


def test_a_first_call_does_not_wait_for_other_streams(ctx):
    """The scratch of a context's first calls with an adapter comes without stopping the device: a host whose other stream is
    busy gets both calls back while it still is."""
    import torch

    from rust_trainer_b200._lib import DT_F32, lib

    L = lib()
    n, k, m, r = 256, 128, 50, 12
    x, dy = (torch.randn(m, c, device="cuda").half() for c in (k, n))

    def calls(c, between=lambda: None):
        packed, _, _, _, f, lin = _make(c, np.random.default_rng(3), Q.Q8_0, n, k, r)
        y, dx = (torch.full((m, cols), float("nan"), device="cuda") for cols in (n, k))
        torch.cuda.synchronize()
        state = between()
        c.check(L.rt_linear_forward_dev(lin._h, x.data_ptr(), m, y.data_ptr(), DT_F32, 0))
        c.check(L.rt_linear_backward_dev(lin._h, x.data_ptr(), dy.data_ptr(), None, m, dx.data_ptr(), 0))
        waited = state is not None and state.query()
        c.synchronize()
        torch.cuda.synchronize()
        g = lin.lora()
        lin.close()
        f.close()
        return waited, [y.cpu().numpy(), dx.cpu().numpy(), g["ga"], g["gb"]]

    def busy():
        side, done = torch.cuda.Stream(), torch.cuda.Event()
        with torch.cuda.stream(side):
            torch.cuda._sleep(1_000_000_000)  # half a second
            done.record(side)
        return done

    _, want = calls(ctx)  # (also loads the kernels)
    c2 = rt.Context(0)
    waited, got = calls(c2, busy)
    assert not waited
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    c2.close()
