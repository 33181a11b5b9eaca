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
# pairs in both directions, and slim pairs in one, where there are pairs
PAIRED = [(Q.Q4_0, 1088, 704, 2600), (Q.Q8_0, 1088, 704, 2600), (Q.Q4_K, 1280, 768, 2500), (Q.Q6_K, 1088, 1280, 2600), (Q.F16, 1088, 1024, 2600)]
SLIM = [(Q.Q6_K, 6400, 256, 130)]


def products(ctx):
    """Results of every case, and the kind of tile of its products: forward and backward."""
    out, kinds = [], []
    for t, n, k, m in CASES + PAIRED + SLIM:
        rng = np.random.default_rng(n + k)
        f = rt.Frozen(ctx, t, n, k, Q.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), t))
        lin = rt.Linear("l", f, rng.standard_normal(n).astype(np.float32))
        lin.attach_lora(16, 32.0, rng.standard_normal((16, k)).astype(np.float32), rng.standard_normal((n, 16)).astype(np.float32))
        x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
        dx = np.zeros((m, k), np.float32)
        f.backward_input(dy, m, dx)
        out += [f.forward(x, m), dx, lin.forward(x, m), lin.backward(x, dy, m)]
        kinds.append([f.tile(m)[0], f.tile(m, True)[0]])
        lin.close()
        f.close()
    return out + [np.array(kinds)]


def test_wide_tiles_give_the_bits_of_pairs(ctx, tmp_path):
    want = products(ctx)
    code = f"import sys; sys.path.insert(0, 'tests'); import numpy as np, rust_trainer_b200 as rt, test_gpu_no_pairs as t; np.savez({str(tmp_path / 'o.npz')!r}, *t.products(rt.Context(0)))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=root, env=dict(os.environ, RT_B200_NO_PAIR="1"))
    got = np.load(tmp_path / "o.npz")
    kinds, without, n = want[-1], got[f"arr_{len(want) - 1}"], len(PAIRED) + len(SLIM)
    assert (kinds[-n:-len(SLIM)] == "pair").all() and (kinds[-len(SLIM):, 1] == "slim").all()
    assert (without[-n:-len(SLIM)] == "wide").all() and not np.isin(without, ["pair", "slim"]).any()
    for i, w in enumerate(want[:-1]):
        assert np.array_equal(got[f"arr_{i}"], w), ((CASES + PAIRED + SLIM)[i // 4], i % 4)
