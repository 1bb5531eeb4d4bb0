"""Rules of the hardware and of the language that the library's sources must keep, read from the sources.

A breach of these is undefined behaviour that timing can hide on every run, so that no result shows it:
they are checked where the code is, without a GPU.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dwim_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
HEADERS = sorted(f for f in os.listdir(CSRC) if f.endswith(".cuh"))

# what reaches another block's shared memory, and what proves that the block is there (ptx.cuh)
REMOTE = re.compile(r"\b(?:st_cluster_f32|ld_cluster_f32|cluster_addr)\s*\(")
MET = re.compile(r"\b(?:cluster_sync|cluster_wait)\s*\(")


def source(name):
    """A source file without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def functions(text):
    """(name, body) of every kernel and device function."""
    for m in re.finditer(r"__global__|__device__ __forceinline__", text):
        at = text.index("{", m.start())
        name = next(n for n in re.findall(r"(\w+)\s*\(", text[m.start():at]) if not n.startswith("__"))
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield name, text[at:end]


def test_every_function_is_found():
    names = [name for f in SOURCES for name, _ in functions(source(f))]
    assert {"normalize_i8_kernel", "matmul_bf16_tile_kernel", "gemm_q4k_kernel", "gemm_dense_kernel", "gemm_few_kernel", "dwim_smallm_kernel",
            "push_shares"} <= set(names)


@pytest.mark.parametrize("name", SOURCES)
def test_a_cluster_meets_before_its_blocks_reach_each_other(name):
    """A block may touch another's shared memory once that block is known to run: after a barrier of the cluster
    (being scheduled together is not having started)."""
    for function, body in functions(source(name)):
        remote = REMOTE.search(body)
        if remote:
            met = MET.search(body)
            assert met and met.start() < remote.start(), f"{function}: a remote access ahead of the cluster's first meeting"


@pytest.mark.parametrize("name", SOURCES + HEADERS)
def test_process_wide_variables_may_be_shared_by_threads(name):
    """Several threads may drive a context each, so what all contexts share is constant, atomic or a thread's own."""
    for m in re.finditer(r"\bstatic\s+((?:[\w:]|<[^<>]*>|\s|\*)+?)\s*\b(\w+)\s*(?:\[[^\]]*\]\s*)*(?:=|;|\{)", source(name)):
        kind = m.group(1)
        assert re.search(r"\b(const|constexpr|thread_local|__device__)\b|\batomic<", kind), f"{name}: static {kind} {m.group(2)}"


def test_a_warpgroup_trades_registers_at_one_instruction():
    """setmaxnreg is for whole warpgroups: all four warps execute the same one.  So it stands first in a branch that
    parts the warps at a multiple of four, ahead of what tells a warpgroup's warps apart; the workers, who take, first."""
    text = "\n".join(source(f) for f in HEADERS + SOURCES)
    numbers = {name: int(value) for name, value in re.findall(r"\b(\w*(?:WARP|WORKERS))\s*=\s*(\d+)\b", text)}
    traders = 0
    for name in SOURCES:
        for function, body in functions(source(name)):
            trades = list(re.finditer(r"\bregs_(dec|inc)\s*<", body))
            if not trades:
                continue
            traders += 1
            assert [m.group(1) for m in trades] == ["inc"] + ["dec"] * (len(trades) - 1), function
            ends = [0]
            for m in trades:
                ahead = re.sub(r"if constexpr \(TRADE\)\s*$", "", body[:m.start()]).rstrip()
                branch = re.search(r"(?:if \(warp < (\w+)\)|else) \{$", ahead)
                assert branch, f"{function}: regs_{m.group(1)} is not the first of a branch for whole warpgroups"
                assert bool(branch.group(1)) == (m is not trades[-1]), function
                ends += [numbers[branch.group(1)]] if branch.group(1) else []
            assert all(e % 4 == 0 for e in ends) and ends == sorted(set(ends)), f"{function}: branches at warps {ends}"
    assert traders == 3


def test_lanes_that_waited_for_several_barriers_meet():
    """A lane that waited for one of several barriers has acquired that one's writes alone, and a warp vote does not order
    memory among lanes: a wait of the whole warp ends at a __syncwarp, on every path."""
    body = dict(functions(source("ptx.cuh")))["mbar_wait_all"]
    assert "return" not in body and re.search(r"__syncwarp\(\);\s*\}$", body)
