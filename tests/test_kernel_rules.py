"""Rules of order that the kernel sources keep and no run shows broken: read from the sources."""
import re
from functools import lru_cache
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "crosspool_b200" / "csrc"
SOURCES = sorted((CSRC / "kernels").glob("*.cu"))


def _plain(text):
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


@lru_cache(maxsize=None)
def functions(path):
    """{name: text of its bodies} of a source or header; bodies inside a function (lambdas) belong to that function."""
    text, out, at = _plain(path.read_text()), {}, 0
    head = re.compile(r"\b([A-Za-z_]\w*)\s*\(([^;{}]|\{\})*\)\s*(?:const\s*)?\{")
    while (m := head.search(text, at)) is not None:
        if m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            inner = re.compile(r"\b([A-Za-z_]\w*)\s*\((?:[^;{}()]|\([^()]*\))*\)\s*\{").search(text, m.start() + len(m.group(1)))
            if m.group(1) != "__launch_bounds__" or inner is None:
                at = m.start() + 1
                continue
            m = inner
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[m.group(1)] = out.get(m.group(1), "") + text[m.end():end]
        at = end
    return out


def _first(pattern, body):
    m = re.search(pattern, body)
    return m.start() if m else None


def test_functions_are_found():
    f = functions(CSRC / "kernels" / "misc.cu")
    assert "map_shared_rank" in f["argmax_kernel"] and "ids[row]" in f["embedding_kernel"] and "pdl::launch" in f["xp_argmax"]
    assert "pdl::release" in functions(CSRC / "kernels" / "gemm_pair.cu")["gemm_pair_kernel"]


@pytest.mark.parametrize("source", SOURCES, ids=lambda p: p.name)
def test_remote_shared_memory_behind_a_cluster_barrier(source):
    """Another CTA's shared memory may be touched once that CTA is known to have started (and its barriers to be initialised)."""
    for name, body in functions(source).items():
        touch = _first(r"\b(map_shared_rank|map_rank|mapa)\b", body)
        if touch is not None:
            met = _first(r"\bcluster_sync\(\)|this_cluster\(\)\s*\.\s*(sync|barrier_wait)\(", body)
            assert met is not None and met < touch, f"{source.name}: {name}"
