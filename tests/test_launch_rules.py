"""Rules of kernels that are launched while the one in front of them still runs (csrc/pdl.cuh), read from the source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "rust_trainer_b200" / "csrc"


def kernels():
    """{name: text of the kernel, from its parameters to the end of its body}, comments taken out."""
    out = {}
    for path in CSRC.glob("*.cu"):
        src = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s+)?(\w+)\(", src):
            at = end = src.index("{", m.end())
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                if depth == 0:
                    break
                end += 1
            out[m[1]] = src[m.end():end]
    return out


@pytest.mark.parametrize("name,when", [
    ("qgemm_kernel", "warp == 2 && (p.late_wait || p.end_wait) && (p.row_scale || (p.residual && OUT != QO_RES))"),
    ("attn_bwd_dq_tc_kernel", "warp == 0")])
def test_what_is_read_without_a_wait_comes_after_an_acquire_fence(name, when):
    """Only the wait is defined to make earlier kernels' writes visible: without it an ordinary load may find an L1 line from
    before them.  One warp's fence in front of the CTA's barrier orders every warp's loads behind it."""
    body = kernels()[name]
    fence = body.index(f"if ({when}) pdl_unwaited();")
    assert body.index("tmem_alloc") < fence < body.index("__syncthreads();", fence) < body.index("tmem_base =")
    for read in ("row_scale[", "lse[", "query_vecs["):
        assert body.find(read) == -1 or body.find(read) > fence
    assert "fence.acq_rel.gpu;" in (CSRC / "pdl.cuh").read_text()


#: kernels that let the next one start before they hold their TMEM, and the layouts of shared memory that keep it free for them
EARLY = {"qgemm_kernel": ("qgemm.cu", r"SMEM_BYTES = SMEM_USED > ALONE_SMEM \? SMEM_USED : ALONE_SMEM;", 1),
         "attn_fwd_tc_kernel": ("attention_tc.cu", r"TOTAL = USED \+ 768 > TWO_BLOCKS_SMEM \? USED \+ 768 : TWO_BLOCKS_SMEM;", 2),
         "attn_bwd_dq_tc_kernel": ("attention_tc.cu", r"TOTAL = USED \+ 768 > TWO_BLOCKS_SMEM \? USED \+ 768 : TWO_BLOCKS_SMEM;", 2)}


@pytest.mark.parametrize("name", sorted(n for n, body in kernels().items() if "tmem_alloc" in body))
def test_no_later_kernel_takes_the_tmem_a_started_one_still_needs(name):
    """Otherwise a CTA of a later kernel on the same SM could take the columns first and wait for this kernel, which waits for
    them."""
    body = kernels()[name]
    assert "pdl_entry" not in body and body.count("pdl_launch_dependents();") == 1
    if body.rindex("tmem_alloc") < body.index("tmem_base =") < body.index("pdl_launch_dependents();"):
        return
    file, layout, times = EARLY[name]
    assert len(re.findall(layout, (CSRC / file).read_text())) == times
    for file, least in (("lowrank_tc.cu", "TOTAL >= LOWRANK_KERNEL_SMEM"), ("lora_grads_tc.cu", "LG_TOTAL >= TMEM_KERNEL_SMEM"),
                        ("attention_tc.cu", "TOTAL >= TMEM_KERNEL_SMEM")):
        assert f"static_assert({least}" in (CSRC / file).read_text()


def test_the_exponents_offset_of_attention_is_fused_by_name():
    """Left to the compiler, a load moved from beside the multiplication to the kernel's front took the fused multiply-add apart: the
    gradients of a 3B step moved by 1e-3."""
    assert re.search(r"off = fmaf\(-my_lse, LOG2E, log2f\(w\) \+ P_BOOST_LOG2\);", kernels()["attn_delta_tc_kernel"])


#: what may be declared __restrict__ in a kernel that starts under the one in front of it: what no kernel of a pass writes (norm
#: weights, biases, tables, what a batch brings along), and results that the kernel only writes
UNWRITTEN = {"w", "qw", "kw", "bias", "cs", "sn", "pos", "idx", "target", "weight", "seq_start", "gap", "tiles"}
ONLY_WRITTEN = {"y16", "out16", "scale", "q16", "k16", "v16", "dq16", "dk16", "dv16", "sq", "sk", "sv", "h", "dg16", "du16", "sg", "su", "d16",
                "logp", "argmax", "lse", "dk", "dv", "dq", "query_vecs", "tops"}
WAITS = sorted(n for n, body in kernels().items() if "pdl_wait();" in body or "pdl_entry();" in body)


@pytest.mark.parametrize("name", WAITS)
def test_what_a_pass_computes_is_read_through_plain_pointers(name):
    """__restrict__ promises that nobody else writes behind the pointer while the kernel runs, which the kernel in front of it still
    does: the compiler may then load before the wait, or through a cache that neither wait nor fence refreshes."""
    body = kernels()[name]
    params = body[:body.index("{")]
    read = {m[1] for m in re.finditer(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)}
    declared = {m[1] for m in re.finditer(r"__restrict__\s+(\w+)", params)}
    assert read <= UNWRITTEN, read - UNWRITTEN
    # (others also read their `out`: a product may be accumulated, a gradient be added where it lies)
    written = ONLY_WRITTEN | ({"out"} if name in ("lowrank_tc_kernel", "gather_f32_rows_kernel") else set())
    assert declared - read <= written, declared - read - written


def test_the_device_word_is_clear_before_a_call_that_reports_an_error_returns():
    """A host that goes on on another stream would otherwise launch kernels that find the old code, give up their waits and, not being
    the first to report, leave the page-locked word at "no error"."""
    src = (CSRC / "api.cu").read_text()
    body = src[src.index("rt_status rt_ctx::check_device_status"):]
    body = body[:body.index("\n}")]
    clear = body.index("cudaMemsetAsync(status_dev, 0")
    assert clear < body.index("cudaStreamSynchronize(stream)", clear) < body.index("return RT_ERR_BAD_INDEX")


@pytest.mark.parametrize("name", ["lowrank_tc_kernel", "lowrank_rows_kernel", "lowrank_rows_many_kernel", "attn_bwd_dkdv_tc_kernel", "lora_grads_tc_kernel"])
def test_a_kernel_with_a_successor_that_reads_unwaited_lets_it_start_after_its_own_wait(name):
    """What is older than such a kernel is then complete when its successor, which reads that without waiting, starts."""
    body = kernels()[name]
    assert "pdl_entry" not in body and body.count("pdl_launch_dependents();") == 1
    assert 0 <= body.index("pdl_wait();") < body.index("pdl_launch_dependents();")


@pytest.mark.parametrize("name", ["lowrank_rows_kernel", "lowrank_rows_many_kernel", "rmsnorm_fwd_lr_kernel", "rmsnorm_bwd_lr_kernel"])
def test_only_prefetches_come_before_the_wait(name):
    body = kernels()[name]
    before = body[body.index("{") + 1:body.index("pdl_wait();")]
    allowed = (r"using C = [^;]*;|constexpr [^;]*;|extern __shared__ [^;]*;|__shared__ [^;]*;|\w+\*? ?\*?\w+ = \(?[\w*]*\)?\(?lr_smem[^;]*;|pdl_launch_dependents\(\);"
               r"|lr_prefetch\([^;]*\);")
    assert re.sub(allowed, "", before).strip() == ""
    prefetch = re.search(r"void lr_prefetch\([^{]*\{(.*?)\n\}", (CSRC / "lowrank_rows.cuh").read_text(), re.S)[1]
    assert "prefetch.global.L2" in prefetch and "ld." not in prefetch and "*(" not in prefetch


def test_row_kernels_with_a_product_are_not_loaded_with_the_others():
    """CUDA loads a file's kernels with the first that is launched, and these are 128 instantiations."""
    assert "_lr_kernel" not in (CSRC / "ops.cu").read_text() and "rmsnorm_fwd_lr_kernel" in kernels()
