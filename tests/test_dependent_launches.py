"""Launches that may be programmatic dependents of the kernel in front (launch_k, launch_k_class of csrc/common.cuh: by their class
or, with FELLM_B200_PDL=1, all of them): the kernel has to wait for that kernel before it touches what it wrote.  Read from the
sources; no GPU."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fellm_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu"))


def closing(text: str, at: int, pair: str) -> int:
    """The index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("brackets do not close")


def source(path: Path) -> str:
    """The file with the sources it includes, without comments."""
    text = path.read_text()
    for inc in re.findall(r'#include\s+"([^"]+\.cu)"', text):
        text += source(CSRC / inc)
    return re.sub(r"//[^\n]*", "", text)


def kernels(text: str):
    """{name: (parameters, body)} of the file's kernels."""
    got = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^;{]*?\)\s*)?(\w+)\s*\(", text):
        end = closing(text, m.end() - 1, "()")
        body = text.index("{", end)
        got[m.group(1)] = (text[m.end():end - 1], text[body:closing(text, body, "{}")])
    return got


def dependents(text: str, names):
    """The kernels that launch_k and launch_k_class are handed: by name, or by the function pointer declared last in front of the call."""
    found = set()
    for m in re.finditer(r"\blaunch_k(?:_class)?\s*\(", text):
        call = text[m.end():closing(text, m.end() - 1, "()")]
        direct = [n for n in names if re.search(rf"\b{n}\b", call)]
        if not direct and re.search(r"\bkern\b", call):
            start = max(text.rfind(decl, 0, m.start()) for decl in ("auto kern", "(*kern)"))
            direct = [n for n in names if re.search(rf"\b{n}\b", text[start:m.start()])]
            assert direct, f"which kernel is launched here? {call[:120]}"
        found.update(direct)
    return found


def waits(name, all_kernels, text, seen=()):
    """Whether the kernel's body, or a device function it calls, waits for the kernel in front."""
    body = all_kernels[name][1]
    if "pdl_wait()" in body:
        return True
    for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\(", body)):
        m = re.search(rf"__device__[^;{{}}]*\b{callee}\s*\(", text)
        if m:
            end = closing(text, m.end() - 1, "()")
            at = text.find("{", end)
            if at >= 0 and "pdl_wait()" in text[at:closing(text, at, "{}")]:
                return True
    return False


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_dependent_kernels_wait(path):
    text = source(path)
    ks = kernels(text)
    launched = dependents(text, ks)
    without = sorted(n for n in launched if not waits(n, ks, text))
    assert not without, f"{path.name}: launched as dependents, but without pdl_wait(): {without}"


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_dependent_kernels_read_the_cache_behind_their_wait(path):
    """A kernel in front may have written into the pool of pages: declared as never changing (const and __restrict__), its loads
    may be moved in front of the wait."""
    text = source(path)
    ks = kernels(text)
    frozen = sorted(n for n in dependents(text, ks) if re.search(r"\bconst\s+\w+\s*\*\s*__restrict__\s+pool\b", ks[n][0]))
    assert not frozen, f"{path.name}: {frozen}"


# What no kernel of a step writes: weights, and the step's index arrays and sampling parameters, which copies from the host bring.
CONSTANT = {"w", "wq", "wc", "wn", "b", "q_w", "k_w", "coef", "table", "Wg", "Wp", "W", "Wr", "corr", "bias", "conv_bias", "freq", "inv_freq", "sinks",
            "positions", "row_slot", "block_table", "item_start", "item_slot", "row_item", "rows", "params", "bias_tok", "bias_val"}
# What kernels only write to.
WRITTEN = {"out", "status", "cq", "lat", "rope", "pool", "q_out", "h", "cast", "y", "out_tokens", "out_probs", "pval", "pidx", "q_abs"}


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_dependent_kernels_read_their_inputs_behind_their_wait(path):
    """Loads through a __restrict__ parameter need not stay behind the wait: nobody else is taken to write there, and where it is const it is
    taken never to change.  So of what a dependent declares __restrict__, no kernel in front writes what it reads."""
    text = source(path)
    ks = kernels(text)
    for name in dependents(text, ks):
        for p in ks[name][0].split(","):
            m = re.search(r"__restrict__\s+(\w+)", p)
            assert not m or m.group(1) in (CONSTANT if re.search(r"\bconst\b[^*]*\*", p) else WRITTEN), \
                f"{path.name}: {name} may read {m.group(1)} ahead of its wait"


def test_the_cache_is_read_ahead_of_a_wait_only_where_the_caller_says_so():
    """latent_tokens_kernel reads index arrays and cache in front of its wait, or waits first: as the caller says.  Who says so has launched
    a product per head in front, an ordinary launch on every route, and writes nothing behind it."""
    text = source(CSRC / "latent_attention_mma.cu")
    body = kernels(text)["latent_tokens_kernel"][1]
    first = body.index("if (!a.ready) pdl_wait();")
    assert all(first < body.index(read) for read in ("a.item_start", "a.positions", "a.block_table", "a.row_slot", "a.pool"))
    assert "launch_k_class(a.ready ? 1 :" in text
    entry = {"fellm_gemm_tiled_batched": ("gemm_tiled", {"gemm_heads_few_kernel", "gemm_tiled_kernel"}),
             "fellm_gemm_simt_batched": ("gemm_simt", {"gemm_tn_simt_kernel"})}
    ops = (CSRC.parent / "ops.py").read_text()
    head_gemm = ops[ops.index("def head_gemm("):ops.index("\n\n\n", ops.index("def head_gemm("))]
    assert set(re.findall(r'"(fellm_\w+)"', head_gemm)) == set(entry)
    for name, (module, launched) in entry.items():
        text = source(CSRC / f"{module}.cu")
        at = text.index(f"{name}(")
        body = text[text.index("{", at):closing(text, text.index("{", at), "{}")]
        assert "launch_k" not in body and "<<<" in body
        assert {k for k in kernels(text) if re.search(rf"\b{k}\b", body)} == launched
    for path in CSRC.parent.rglob("*.py"):
        text = path.read_text()
        for m in re.finditer(r"cache_ready=True", text):
            call = text.rindex("ops.latent_attention(", 0, m.start())
            product = text.rindex("ops.head_gemm(", 0, call)
            assert set(re.findall(r"\bops\.(\w+)\(", text[product:call])) <= {"head_gemm", "latent_rotate_q"}, path


def test_the_reading_finds_the_launches():
    """(the checks above would pass on files they cannot read)"""
    found = {p.stem: dependents(source(p), kernels(source(p))) for p in SOURCES}
    assert sum(len(v) for v in found.values()) > 40
    assert "rmsnorm_vec_kernel" in found["elementwise"] and "attention_prefill_umma_kernel" in found["attention_umma"]
    assert "latent_gather_kernel" in found["latent"] and "gemm_tiled_kernel" not in found["gemm_tiled"]
