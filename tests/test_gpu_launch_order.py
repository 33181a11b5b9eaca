"""Kernels that start beside the one in front of them (csrc/pdl.cuh) give the bits of strict stream order (RT_B200_PDL=0): with the
rule by size, and with programmatic launches at every size (RT_B200_PDL=1)."""
import os
import subprocess
import sys

import numpy as np
import pytest

import rust_trainer_b200 as rt
from rust_trainer_b200 import quants as Q
from rust_trainer_b200 import synth

pytestmark = pytest.mark.gpu
# preset, quant, rank, sequence lengths: below and above the 4096 tokens up to which launches are programmatic
STEPS = [("tiny-qwen3", "Q4_0", 8, [64] * 4), ("tiny-qwen3", "Q8_0", 12, [900] * 5), ("tiny-qwen2", "Q8_0", 16, [130, 77, 700]),
         ("tiny-qwen3-hd128", "Q4_0", 16, [256] * 4), ("tiny-qwen3-hd128", "Q8_0", 16, [1100] * 4), ("tiny-llama", "Q8_0", 16, [515, 33])]


def results(ctx):
    out = []
    for preset, quant, rank, lens in STEPS:
        spec = synth.preset(preset, quant=quant, seed=5, w_std=0.05)
        gm = rt.Model(ctx, spec.config(), synth.build_tensors(spec))
        gm.attach_lora(rank, 2.0 * rank, None, 1)
        gm.load_adapters(synth.lora_adapters(spec, rank, 2.0 * rank, seed=7, b_std=0.02))
        seqs = [synth.token_batch(spec, 1, n, 11 + i)[0] for i, n in enumerate(lens)]
        parts = [synth.answer_targets(s, s.size // 2) for s in seqs]
        at = np.cumsum([0] + lens[:-1])
        tp, tt = np.concatenate([p[0] + a for p, a in zip(parts, at)]), np.concatenate([p[1] for p in parts])
        w = np.full(tp.size, 1.0 / tp.size, np.float32)
        for _ in range(3):  # eager, captured, replayed
            gm.zero_grad()
            out.append(gm.forward_backward(seqs, tp, tt, w)[0].copy())
            out.append(np.concatenate([np.concatenate([g["ga"].ravel(), g["gb"].ravel()]) for g in (l.lora() for l in gm.lora_linears())]))
        gm.close()
    for t, n, k, m in [(Q.Q8_0, 3072, 1024, 700), (Q.F16, 1088, 704, 33), (Q.Q6_K, 512, 1024, 5000)]:
        rng = np.random.default_rng(n)
        f = rt.Frozen(ctx, t, n, k, Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t))
        lin = rt.Linear("l", f, rng.standard_normal(n).astype(np.float32))
        lin.attach_lora(12, 24.0, rng.standard_normal((12, k)).astype(np.float32), rng.standard_normal((n, 12)).astype(np.float32))
        x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
        dx = np.zeros((m, k), np.float32)
        f.backward_input(dy, m, dx)
        out += [f.forward(x, m), dx, lin.forward(x, m), lin.backward(x, dy, m), lin.lora()["ga"], lin.lora()["gb"]]
        lin.close()
        f.close()
    return out


def test_overlapped_launches_give_the_bits_of_strict_order(ctx, tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = {}
    for pdl in ("0", "1", ""):
        path = str(tmp_path / f"o{pdl}.npz")
        code = f"import sys; sys.path.insert(0, 'tests'); import numpy as np, rust_trainer_b200 as rt, test_gpu_launch_order as t; np.savez({path!r}, *t.results(rt.Context(0)))"
        env = {k: v for k, v in os.environ.items() if k != "RT_B200_PDL"}
        subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=root, env=dict(env, RT_B200_PDL=pdl) if pdl else env)
        got[pdl] = np.load(path)
    for name in got["0"].files:
        assert np.isfinite(got["0"][name]).all()
        assert np.array_equal(got["1"][name], got["0"][name]) and np.array_equal(got[""][name], got["0"][name]), name
