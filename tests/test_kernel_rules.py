"""Rules of order that the kernel sources keep and no run shows broken: read from the sources."""
import re
from functools import lru_cache
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "crosspool_b200" / "csrc"
SOURCES = sorted((CSRC / "kernels").glob("*.cu"))


def _plain(text):
    """The text without comments and launch bounds."""
    text = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))
    return re.sub(r"__(launch_bounds|maxnreg)__\s*\([^()]*\)", "", text)


@lru_cache(maxsize=None)
def functions(path):
    """{name: text of its bodies} of a source or header; bodies inside a function (lambdas) belong to that function."""
    text, out, at = _plain(path.read_text()), {}, 0
    head = re.compile(r"\b([A-Za-z_]\w*)\s*\(([^;{}]|\{\})*\)\s*(?:const\s*)?\{")
    while (m := head.search(text, at)) is not None:
        if m.group(1) in ("if", "for", "while", "switch"):
            at = m.start() + 1
            continue
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


# ---------------------------------------------------------------- kernels that start before their predecessor ends (pdl.cuh)


def _all_functions():
    out = {}
    for p in [*SOURCES, *sorted((CSRC / "include" / "xpool").glob("*.cuh"))]:
        for name, body in functions(p).items():
            out.setdefault(name, []).append((p, body))
    return out


def dependent_kernels(source):
    text = _plain(source.read_text())
    launched = re.findall(r"pdl::launch\(([^,]*),", text)
    if any(arg.strip() == "kernel" for arg in launched):      # chosen in front of the launch, or handed to a lambda that launches it
        launched += re.findall(r"auto kernel =([^;]*);|\bgo\(([^;]*), p\);", text)
        launched = ["".join(arg) for arg in launched]
    return sorted({k for arg in launched for k in re.findall(r"\b\w+_kernel\b", arg)})


def _reached(source, kernel):
    """Bodies of a kernel and of what it calls, from its own file or from headers."""
    every, seen, todo = _all_functions(), {}, [kernel]
    while todo:
        name = todo.pop()
        if name in seen or name not in every:
            continue
        seen[name] = "".join(b for p, b in every[name] if p == source or p.suffix == ".cuh")
        todo += re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^<>;]*>)?\s*\(", seen[name])
    return seen


DEPENDENT = [pytest.param(s, k, id=f"{s.stem}-{k}") for s in SOURCES for k in dependent_kernels(s)]


def test_dependent_kernels_are_found():
    assert {"gemm_ws_kernel", "gemm_pair_kernel", "gemm_stream_kernel", "argmax_kernel", "norm_rows_kernel", "rope_kv_kernel", "combine_kernel",
            "prefill_attn_umma_kernel", "decode_attn_tc_kernel", "resid_norm_kernel", "latent_prep_kernel"} <= {p.values[1] for p in DEPENDENT}


@pytest.mark.parametrize("source,kernel", DEPENDENT)
def test_early_kernels_read_nothing_through_the_non_coherent_path(source, kernel):
    """Such loads are for data that nobody writes while the kernel runs; these kernels run while the one before them may still write."""
    for name, body in _reached(source, kernel).items():
        assert re.search(r"ld\.global\.nc|\b__ldg\(", body) is None, f"{kernel}: {name}"
    text = _plain(source.read_text())
    for m in re.finditer(rf"\b{kernel}\(([^)]*)\)\s*\{{", text):
        assert "__restrict__" not in m.group(1), kernel


@pytest.mark.parametrize("source,kernel", DEPENDENT)
def test_early_kernels_wait_before_they_let_the_next_one_start(source, kernel):
    bodies = [b for b in _reached(source, kernel).values() if "pdl::" in b]
    assert bodies, f"{kernel} never waits for its predecessor"
    for body in bodies:
        wait, release = _first(r"pdl::wait\(\)", body), _first(r"pdl::release(_short)?\(\)", body)
        assert wait is not None and (release is None or wait < release), kernel


@pytest.mark.parametrize("source,kernel", DEPENDENT)
def test_kernels_that_handshake_with_other_gpus_do_not_start_early(source, kernel):
    for name, body in _reached(source, kernel).items():
        assert re.search(r"\b(wait_flag_ge|st_release_sys|ld_acquire_sys)\(", body) is None, f"{kernel}: {name}"
