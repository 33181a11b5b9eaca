"""Where CTA pairs cannot run, or are switched off, the wide single-CTA tiles take their place: the same bits."""
import os
import subprocess
import sys

import numpy as np
import pytest

import rust_trainer_b200 as rt
from rust_trainer_b200 import quants as Q

pytestmark = pytest.mark.gpu
CASES = [(Q.Q4_0, 320, 704, 2600), (Q.Q8_0, 1088, 704, 300), (Q.Q4_K, 192, 768, 2600), (Q.Q6_K, 1088, 768, 1300), (Q.F16, 320, 704, 2600), (Q.BF16, 256, 704, 97)]


def products(ctx):
    out = []
    for t, n, k, m in CASES:
        rng = np.random.default_rng(n + k)
        f = rt.Frozen(ctx, t, n, k, Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t))
        lin = rt.Linear("l", f, rng.standard_normal(n).astype(np.float32))
        lin.attach_lora(16, 32.0, rng.standard_normal((16, k)).astype(np.float32), rng.standard_normal((n, 16)).astype(np.float32))
        x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
        dx = np.zeros((m, k), np.float32)
        f.backward_input(dy, m, dx)
        out += [f.forward(x, m), dx, lin.forward(x, m), lin.backward(x, dy, m)]
        lin.close()
        f.close()
    return out


def test_wide_tiles_give_the_bits_of_pairs(ctx, tmp_path):
    want = products(ctx)
    code = f"import sys; sys.path.insert(0, 'tests'); import numpy as np, rust_trainer_b200 as rt, test_gpu_no_pairs as t; np.savez({str(tmp_path / 'o.npz')!r}, *t.products(rt.Context(0)))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=root, env=dict(os.environ, RT_B200_NO_PAIR="1"))
    got = np.load(tmp_path / "o.npz")
    for i, w in enumerate(want):
        assert np.array_equal(got[f"arr_{i}"], w), (CASES[i // 4], i % 4)
