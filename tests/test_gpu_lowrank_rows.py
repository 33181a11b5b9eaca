"""The adapters' low-rank products inside the RMSNorm kernels and over rows in memory (csrc/lowrank_rows.cuh): every group count of
rank indices, row lengths with full and ragged shares of K, batches that end inside a group of eight tokens, and both forms of each
kernel (up to 2048 tokens and beyond) against each other."""
import numpy as np
import pytest

import rust_trainer_b200 as rt
from conftest import cosine, rel_l2
from oracle import oracle as O
from rust_trainer_b200 import quants as Q
from rust_trainer_b200 import synth
from test_gpu_model import GRAD_COS, GRAD_TOL, LOSS_TOL, _batch, _flat, _gpu_flat, _oracle_step

pytestmark = pytest.mark.gpu


def _spec(hidden, seed=5):
    return synth.preset("tiny-qwen3", quant="Q8_0", seed=seed, w_std=0.05, hidden=hidden)


def _model(ctx, spec, rank):
    tensors = synth.build_tensors(spec)
    synth.perturb_norms(tensors, 7)
    ads = synth.lora_adapters(spec, rank, 2.0 * rank, seed=9, b_std=0.02)
    gm = rt.Model(ctx, spec.config(), tensors)
    gm.attach_lora(rank, 2.0 * rank, None, 1)
    gm.load_adapters(ads)
    return tensors, ads, gm


# hidden sizes: one block of K per warp and fewer, 28 blocks on eight warps, the widest; ranks: 1 to 64 of a linear, 24 to 64 of a stack
@pytest.mark.parametrize("hidden,rank,lens", [(128, 8, [1 + 8]), (384, 1, [7, 2]), (640, 24, [17]), (896, 16, [70, 3]), (1024, 32, [33, 8]),
                                              (1024, 64, [5, 60]), (256, 40, [41])])
def test_gradients_match_the_oracle(ctx, hidden, rank, lens):
    spec = _spec(hidden)
    tensors, ads, gm = _model(ctx, spec, rank)
    om = O.OracleModel(spec.config(), tensors)
    om.attach_lora(ads)
    seqs, tp, tt, per_seq = _batch(spec, lens, seed=11)
    w = np.full(tp.size, 1.0 / tp.size, np.float32)
    lp_o = _oracle_step(om, seqs, per_seq, w)
    gm.zero_grad()
    lp_g, _ = gm.forward_backward(seqs, tp, tt, w)
    assert np.max(np.abs(lp_g - lp_o) / np.abs(lp_o)) < LOSS_TOL
    go, gg = _flat(om.lora, "ga", "gb"), _gpu_flat(gm, "ga", "gb")
    assert rel_l2(gg, go) < GRAD_TOL and cosine(gg, go) > GRAD_COS
    for lin, e in zip(gm.lora_linears(), om.lora):
        g = lin.lora()
        assert cosine(np.concatenate([g["ga"].ravel(), g["gb"].ravel()]), np.concatenate([e["ga"].ravel(), e["gb"].ravel()])) > GRAD_COS
    gm.close()
    om.close()


# widths and ranks of every form beyond 2048 tokens: forward products of one to four groups of rank indices (stacks of two and three
# adapters of up to 20), backward ones of one to four
@pytest.mark.parametrize("hidden,rank", [(256, 4), (1024, 16), (896, 20), (640, 12), (384, 40), (128, 64)])
def test_a_sequence_gets_the_same_products_in_a_small_and_a_large_batch(ctx, hidden, rank):
    """Two sequences alone, and as the first and the last of a batch of 9347 tokens: persistent CTAs take two to eight groups of rows
    in turn (at most two of an SM, with eight or sixteen rows each: 4736 tokens at a time), and the last group is not full."""
    spec = _spec(hidden)
    _, _, gm = _model(ctx, spec, rank)
    fill = list(synth.token_batch(spec, 71, 128, 3))
    ends = [synth.token_batch(spec, 1, n, 5 + n)[0] for n in (128, 131)]
    parts = [synth.answer_targets(q, 64) for q in ends]

    def run(seqs, tp, tt, w):
        gm.zero_grad()
        lp, _ = gm.forward_backward(seqs, tp, tt, w)
        return lp, _gpu_flat(gm, "ga", "gb")

    def weights(n):
        return np.full(n, 1.0 / 64, np.float32)

    alone = [run([q], p, t, weights(p.size)) for q, (p, t) in zip(ends, parts)]
    lead = 128 * (1 + len(fill))  # (sequences that start on a tile boundary)
    idle = np.arange(128, lead - 1, 97)
    tp = np.concatenate([parts[0][0], idle, parts[1][0] + lead])
    tt = np.concatenate([parts[0][1], 0 * idle, parts[1][1]])
    w = np.concatenate([weights(parts[0][0].size), np.zeros(idle.size, np.float32), weights(parts[1][0].size)])
    lp, grads = run([ends[0], *fill, ends[1]], tp, tt, w)
    assert np.array_equal(alone[0][0], lp[:parts[0][0].size]) and np.array_equal(alone[1][0], lp[-parts[1][0].size:])
    # the gradients' last f32 sums (over key tiles, over splits of tokens, over the two sequences) fall differently, a few 2^-24; another
    # rounding of a 16-bit product anywhere would show as 2^-12 of its value
    assert rel_l2(grads, alone[0][1] + alone[1][1]) < 1e-6 and all(np.abs(g).max() > 0 for _, g in alone)
    gm.close()


@pytest.mark.parametrize("hidden,rank,lens", [(128, 16, [128, 77]), (128, 8, [900] * 4), (384, 20, [205]), (896, 8, [70, 3]), (1024, 32, [300])])
def test_recomputed_blocks_get_the_bits_of_kept_ones(ctx, hidden, rank, lens):
    """A block's second forward keeps Hs and takes RMSNorm without the product: the same rows all the same."""
    spec = synth.preset("tiny-qwen3", quant="Q8_0", seed=5, w_std=0.05, hidden=hidden, n_layers=4)
    _, _, gm = _model(ctx, spec, rank)
    seqs, tp, tt, _ = _batch(spec, lens, seed=11)
    w = np.full(tp.size, 1.0 / tp.size, np.float32)
    got = []
    for mode in (0, 1):
        gm.set_checkpointing(mode)
        gm.zero_grad()
        gm.forward_backward(seqs, tp, tt, w)
        got.append(_gpu_flat(gm, "ga", "gb"))
    assert np.array_equal(*got) and np.abs(got[0]).max() > 0
    gm.close()


def test_only_a_pass_with_active_adapters_asks_for_their_scratch():
    """Scoring with the base model (no adapter enabled) leaves Hs' memory, 128 bytes a token, unasked for."""
    import torch

    c = rt.Context(0)
    spec = _spec(256)
    _, _, gm = _model(c, spec, 8)
    toks = synth.token_batch(spec, 64, 1024, 3)
    tp, tt = synth.answer_targets(toks[0], 64)

    def free_after_a_pass():
        gm.score(list(toks), tp, tt)
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    gm.set_lora_enabled(False)
    base = free_after_a_pass()
    gm.set_lora_enabled(True)
    assert base - free_after_a_pass() >= 64 * 1024 * 64 * 2
    gm.close()
    c.close()


# columns: one block of K for one warp, a ragged share of the second block, all of it; tokens: just beyond what the GPU holds at a
# time, ragged last groups, several rounds
@pytest.mark.parametrize("k,r,m", [(32, 1, 4737), (544, 3, 9475), (896, 16, 16391), (1024, 8, 30001)])
def test_products_of_many_tokens(ctx, k, r, m):
    """A linear whose weights are zero gives the adapter alone: the reference's value, and the bits of the same tokens in batches
    small enough for the other kernel."""
    rng = np.random.default_rng(m)
    n = 64
    f = rt.Frozen.from_f32(ctx, np.zeros((n, k), np.float32), Q.Q8_0)
    lin = rt.Linear("l", f)
    a, b = rng.standard_normal((r, k)).astype(np.float32), rng.standard_normal((n, r)).astype(np.float32)
    lin.attach_lora(r, 2.0 * r, a, b)
    x = rng.standard_normal((m, k)).astype(np.float32)
    y = lin.forward(x, m)
    # x, s A, the product and B are rounded to f16, 2^-12 of each value on average at most, and the sums are f32
    want = 2.0 * (x.astype(np.float64) @ a.T.astype(np.float64)) @ b.T.astype(np.float64)
    assert rel_l2(y, want) < 4 * 2.0 ** -12
    parts = [lin.forward(x[i:i + 4096], min(4096, m - i)) for i in range(0, m, 4096)]
    assert np.array_equal(y, np.concatenate(parts))
    lin.close()
    f.close()
