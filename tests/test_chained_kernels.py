"""The start of kernels that begin while the one before them drains, checked in their source."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "shardtrain_b200" / "csrc"


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
