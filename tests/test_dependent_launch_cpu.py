"""Kernels start before the launch ahead of them is through, so what that launch writes is loaded behind the dependency wait.  The
compiler keeps a load there unless it is told that nobody writes the memory: const __restrict__ parameters, __ldg and
ld.global.nc stand for weights, tables and descriptors alone."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "runnburn_b200" / "csrc"
FILES = sorted(p for p in CSRC.glob("*") if p.suffix in (".cuh", ".cu", ".inc", ".hpp"))
# what no launch of a chain writes: weights and biases, decays, embedding and rotation tables, tensor maps, the list of peers
CONSTANTS = {"w", "w0", "w2", "b", "uv", "decay", "table", "rope_table", "tmaps", "peers"}
# the weights' bytes and rows that read-only loads take, as the kernels write them
READ_ONLY_LOADS = {
    "common.cuh": {"c_exp2_tab32 + i"},
    "dense.cuh": {"w0 + k", "w1 + k"},
    "gemv_stream.cuh": {"w + k", "w + k + 1"},
    "latent_attention.cuh": {"w + (size_t)i * d.rank", "w + e"},
    "linear_state.cuh": {"a.w2 + ((size_t)h * dim + dch) * a.rank + dl * seg + i * 8", "a.w2 + ((size_t)h * dim + ch) * a.rank + dl * seg + i * 8"},
    "moe.cuh": {"wr + u * 16 + j", "wr + base + 16 * WB + u * 16 + j"},
    "prefill_gemm.cuh": {"base + 16 * j"},
    "prefill_gemm_split.cuh": {"blk + 8 * h", "blk + 16 + 32 * g + 16 * h"},
    "q8k.cuh": {"reinterpret_cast<const float4 *>(w + b * 256 + lane * 8)", "reinterpret_cast<const float4 *>(w + b * 256 + lane * 8 + 4)"},
}


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def arguments(text, call):
    """The text between the parentheses of every call."""
    for m in re.finditer(rf"(?<![\w.]){call}\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_restrict_is_for_what_no_launch_writes(path):
    for m in re.finditer(r"([\w:<> ]*[\w>] ?\*(?:const \*)?)__restrict__ (\w+)", code(path)):
        assert "const" in m.group(1) and m.group(2) in CONSTANTS, m.group(0)
    assert len(re.findall("__restrict__", code(path))) == len(re.findall(r"\*(?:const \*)?__restrict__ \w", code(path)))


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_read_only_loads_are_of_weights(path):
    text = code(path)
    if path.name == "common.cuh":   # the loads themselves
        text = re.sub(r"__device__[^;{]*ldg_nc_u\d\([^)]*\) \{", "", text)
        assert text.count("ld.global.nc") == 2
    else:
        assert "ld.global.nc" not in text
    found = {a for call in ("__ldg", "ldg_nc_u2", "ldg_nc_u4") for a in arguments(text, call)}
    assert found <= READ_ONLY_LOADS.get(path.name, set()), found


@pytest.mark.parametrize("path", FILES, ids=lambda p: p.name)
def test_loads_from_l2_keep_their_place(path):
    """ld_l2 stays behind waits and fences; the built-in promises nothing of the kind."""
    assert not re.search(r"__ldc[gas]\(", code(path))
