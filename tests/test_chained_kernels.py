"""Kernels that start while their predecessor still writes (csrc/common.cuh: chain_wait), checked in their
source: what a predecessor may write is not declared `__restrict__` nor loaded through the read-only path,
since both allow the compiler to read it before the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "shardtrain_b200" / "csrc"
# what no kernel of a chain writes
CONSTANT = {"w", "cos_t", "sin_t", "positions"}


def functions(text):
    """(name, parameters, body) of the kernels and device functions."""
    head = re.compile(r"(?:__global__|__device__)[^;{}()]*?(?:__launch_bounds__\([^)]*\)|__cluster_dims__\([^)]*\)|[^;{}()])*?"
                      r"\b(\w+)\(((?:[^(){};]|\([^()]*\))*)\)\s*\{")
    for match in head.finditer(text):
        depth, end = 1, match.end()
        while depth:
            depth += (text[end] == "{") - (text[end] == "}")
            end += 1
        yield match.group(1), match.group(2), text[match.end():end]


def chained():
    """The functions that wait for a predecessor, and the kernels that consist of such a function."""
    found = [f for path in sorted(CSRC.glob("*.cu*")) for f in functions(path.read_text())]
    waiting = {name for name, _, body in found if "chain_wait();" in body}
    return [f for f in found if f[0] in waiting
            or any(re.search(rf"\b{name}\s*[<(]", f[2]) for name in waiting if name.endswith("_body"))]


def test_the_chained_kernels_are_found():
    names = {name for name, _, _ in chained()}
    assert {"rmsnorm_fwd_kernel", "rmsnorm_bwd_kernel", "rmsnorm_bwd_rows_kernel", "colsum_f32_kernel",
            "colsum_bf16_partial_kernel", "rope_kernel", "swiglu_bwd_kernel", "cast_f32_bf16_kernel",
            "attention_fwd_kernel", "attention_delta_kernel", "attention_dq_kernel", "attention_dkv_kernel",
            "attention_dkv_finish_kernel", "gemm_bf16_tcgen05_kernel", "gemm_pair_bf16_tcgen05_kernel",
            "gemm_bf16_tcgen05_body"} <= names


def test_what_a_predecessor_writes_is_not_restrict():
    for name, parameters, body in chained():
        qualified = set(re.findall(r"__restrict__\s+(\w+)", parameters + body))
        assert qualified <= CONSTANT, (name, qualified - CONSTANT)


def test_what_a_predecessor_writes_is_not_read_through_the_read_only_path():
    for name, _, body in chained():
        for use in re.findall(r"__ldg\(([^;]*)\)", body):
            assert use.startswith("ep.bias"), (name, use)        # a weight
        assert ".nc." not in body, name


def test_a_pair_meets_before_it_allocates_tmem_together():
    """An allocation for two CTAs is carried out by both: each knows that the other runs."""
    found = [body for path in sorted(CSRC.glob("*.cu*")) for _, _, body in functions(path.read_text())
             if "tmem_alloc_pair(" in body]
    assert found
    for body in found:
        before = body[:body.index("tmem_alloc_pair(")]
        meeting = before.rindex("cluster_sync();")
        # and nothing of the pair is asked for in between
        assert not re.search(r"st_cluster\(|peer_word\(|_pair\(", before[:meeting])
