"""Bounded waits of the kernels, read from their sources: no GPU is made to run out of one."""

import os
import re

import pytest

from servelab_b200.csrc import build

CSRC = os.path.dirname(build.__file__)
# kernels whose roles go on with instructions that a whole warp executes (elections, shuffles, tensor memory)
WARP_KERNELS = ["attention_tc.cu", "attention_kv_tc.cu", "attention_decode.cu", "gemm_rows.cu", "gemm_tcgen05.cu"]


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, at):
    """The braces' contents from the first brace behind ``at`` on."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("no closing brace")


def test_the_list_is_complete():
    elected = [n for n in sorted(os.listdir(CSRC)) if n.endswith(".cu") and "slb_elected()" in source(n)]
    assert set(elected) <= set(WARP_KERNELS)


@pytest.mark.parametrize("name", WARP_KERNELS)
def test_a_warp_gives_a_wait_up_as_one(name):
    """A bound that runs out in some lanes only must not part them from the others, who would wait for them at the next
    election or shuffle: the outcome of every wait is voted on, in the wait or around its call."""
    text = source(name)
    voted, plain = set(), {"mbar_wait"}                    # (mbar_wait of mma_util.cuh is a single thread's)
    for m in re.finditer(r"__device__ __forceinline__ bool (\w+)\(uint64_t\* bar, uint32_t parity\)", text):
        if re.search(r"return slb_warp_agrees\(done != 0\);\s*}$", body(text, m.end())):
            assert body(text, m.end()).count("return") == 1
            voted.add(m.group(1))
        else:
            plain.add(m.group(1))
    plain -= voted
    for m in re.finditer(r"\b(%s)\(&?\w" % "|".join(plain), text) if plain else ():
        before = text[max(0, m.start() - 200):m.end()]
        assert ("slb_warp_agrees(" + m.group(1) in before
                or re.search(r"if \(tid == 0\)\s+for [^\n]*\s+\w+\(&\w$", before)), m.group(0)
    assert voted or "slb_warp_agrees(mbar_wait" in text


@pytest.mark.parametrize("name", ["attention_tc.cu", "attention_kv_tc.cu", "gemm_rows.cu", "gemm_tcgen05.cu"])
def test_a_loader_waits_for_the_copies_it_has_asked_for(name):
    """Whichever role gives up, the block must not leave while copies into its shared memory are in flight: every loader ends
    with a bounded wait for the last copy of each stage, on no condition but being the one that counts them."""
    text = source(name)
    loops = [m for m in re.finditer(r"if \(!mbar_wait\(&(?:empty|freed)\[\w+\]", text)]
    ends = list(re.finditer(r"(if \(rank == 0\)\s*)?for \((?:int|uint32_t) \w+ = (?:max\(0, asked - \w+\)|it > [^;]*); \w+ < (?:asked|it); \+\+\w+\)"
                            r"\s*mbar_wait\(&full\[", text))
    assert len(loops) == len(ends) == (2 if name == "gemm_tcgen05.cu" else 1)
    for a, b in zip(loops, ends):
        assert a.start() < b.start() and "!ok" not in text[b.start() - 80:b.start()]


def test_a_cluster_whose_block_gave_up_stores_nothing():
    """Blocks that share a tile's keys add their parts up: with one part missing the sum is no result.  The block that gave
    up says so in a word of its own (not by the numbers of its part, which a block without keys leaves as well), every block
    of the cluster reads all words behind the barrier, and stores only where none is set."""
    text = source("attention_tc.cu")
    assert re.search(r"mbar_init\(q_full, 1\);\s*\*reinterpret_cast<volatile int\*>\(smem \+ OFF_GAVE\) = 0;", text)
    assert "if (!ok) *reinterpret_cast<volatile int*>(smem + OFF_GAVE) = 1;" in text
    combine = text[text.index("if (splits > 1) {\n        __syncwarp();"):]
    combine = combine[:combine.index("tcgen05.dealloc")]
    assert re.search(r"for \(int k = 0; k < splits; \+\+k\) \{[^}]*whole = whole && [^;]*OFF_GAVE\), k\)\) == 0;", combine)
    stores = [m.start() for m in re.finditer(r"reinterpret_cast<uint4\*>\(dst", combine)]
    assert len(stores) == 1 and combine.index("if (whole && r < nrows) {") < stores[0]


@pytest.mark.parametrize("path", ["bench.py", os.path.join("servelab_b200", "bench", "kernel_bench.py")])
def test_benchmarks_read_the_status_of_every_kernel_they_run(path):
    """A run counts as clean by these words: the products of a prompt's feed-forward are among them."""
    with open(os.path.join(os.path.dirname(os.path.dirname(CSRC)), path)) as f:
        words = re.search(r"status = (\{.*?\})", f.read(), re.S).group(1)
    for call in ("gemm_tc_status()", "gemm_rows_status()", "attention_status(", "prefill_attention_tc_status(",
                 "decode_attention_status("):
        assert "K." + call in words


def test_the_vote_is_of_all_lanes():
    text = source("common.cuh")
    assert "__all_sync(0xffffffffu, seen)" in body(text, text.index("bool slb_warp_agrees("))
