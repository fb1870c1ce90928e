"""The waits of the warps that issue the float32 products (csrc/ring_turns.h, used by csrc/linear_f32_split.cu), walked through every
order in which copies may land, products end, barriers be told of it and warps run: nobody starts a k block whose stage is not filled
or whose sum is not drained, and nobody waits for good."""

import os
import shutil
import subprocess

import pytest

import ullm_b200.csrc.build as build

BLOCKS = 8
EMPTY, FULL, SUM = 0, 1, 2

PROGRAM = """
#include <cstdio>
#include "ring_turns.h"
int main() {
  const int rings[4][2] = {{3, 4}, {3, 2}, {2, 4}, {2, 2}};
  for (auto& r : rings)
    for (int kb = 0; kb < %d; ++kb) {
      std::printf("%%d %%d %%d", r[0], r[1], kb);
      ring_issue_turn(kb, r[0], r[1], [](RingBarrier which, int i, unsigned parity) { std::printf(" %%d %%d %%u", (int)which, i, parity); return true; });
      std::printf("\\n");
    }
}
""" % BLOCKS


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    """{(stages, sums): [the waits of block 0, of block 1, ..]} as the header gives them."""
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    work = tmp_path_factory.mktemp("turns")
    (work / "turns.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", build.HERE, str(work / "turns.cpp"), "-o", str(work / "turns")], check=True)
    out = {}
    for line in subprocess.run([str(work / "turns")], check=True, capture_output=True, text=True).stdout.splitlines():
        stages, sums, _, *waits = map(int, line.split())
        out.setdefault((stages, sums), []).append([tuple(waits[i:i + 3]) for i in range(0, len(waits), 3)])
    return out


def walk(turns, stages, sums, issuers):
    """Every state that can be reached; what goes wrong in one of them, or None.

    The state: k blocks split (stored) and, for the block being split, nothing more; blocks whose copies are on their way; per issuing
    warp its block and the next of its waits; blocks whose products run, with the two barriers that are still to be told; blocks drained.
    A barrier is the number of its completed phases (the splitting warps count as one: they run in order and arrive once per block)."""
    start = (0, frozenset(), tuple((w, 0) for w in range(issuers)), frozenset(), frozenset(), 0)
    seen, todo = {start}, [start]
    while todo:
        split, flying, warps, telling_stage, telling_sum, drained = state = todo.pop()
        issued = {b for w, (at, _) in enumerate(warps) for b in range(w, at, issuers)}
        stage_told, sum_told = issued - telling_stage, issued - telling_sum

        # completed phases: a stage's `full` needs its blocks split and landed, one after the other (a later one cannot begin before)
        def phases(ring, done):
            n = {}
            for b in range(BLOCKS):
                if b in done:
                    n[b % ring] = n.get(b % ring, 0) + 1
            return n

        full = phases(stages, {b for b in range(split) if b not in flying})
        empty, sum_full = phases(stages, stage_told), phases(sums, sum_told)
        sum_empty = phases(sums, set(range(drained)))

        def passes(phase_count, parity):
            return (phase_count & 1) != parity

        nxt = []
        if split < BLOCKS and empty.get(split % stages, 0) >= split // stages:  # (waits for this stage's uses in order: exact)
            nxt.append((split + 1, flying | {split}, warps, telling_stage, telling_sum, drained))
        for b in flying:  # (any order)
            nxt.append((split, flying - {b}, warps, telling_stage, telling_sum, drained))
        for w, (kb, i) in enumerate(warps):
            if kb >= BLOCKS:
                continue
            waits = turns[kb]
            if i < len(waits):
                which, index, parity = waits[i]
                if passes({EMPTY: empty, FULL: full, SUM: sum_empty}[which].get(index, 0), parity):
                    nxt.append((split, flying, warps[:w] + ((kb, i + 1),) + warps[w + 1:], telling_stage, telling_sum, drained))
                continue
            if not kb < split or kb in flying:
                return f"block {kb} begins before its stage is filled"
            if drained < kb - sums + 1:
                return f"block {kb} begins before its sum is drained"
            nxt.append((split, flying, warps[:w] + ((kb + issuers, 0),) + warps[w + 1:], telling_stage | {kb}, telling_sum | {kb}, drained))
        for b in telling_stage:
            nxt.append((split, flying, warps, telling_stage - {b}, telling_sum, drained))
        for b in telling_sum:
            nxt.append((split, flying, warps, telling_stage, telling_sum - {b}, drained))
        if drained < BLOCKS and sum_full.get(drained % sums, 0) > drained // sums:
            nxt.append((split, flying, warps, telling_stage, telling_sum, drained + 1))
        if not nxt and drained < BLOCKS:
            return f"everyone waits with {drained} blocks drained: {state}"
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("stages,sums", [(3, 4), (3, 2), (2, 4), (2, 2)])
@pytest.mark.parametrize("issuers", [1, 2])
def test_no_block_begins_early_and_none_is_forgotten(turns, stages, sums, issuers):
    assert walk(turns[stages, sums], stages, sums, issuers) is None


def test_the_wait_for_a_full_stage_alone_mistakes_an_old_use(turns):
    """What the walk is for: without the wait for the stage to be given back, two warps and three stages go wrong."""
    alone = [[w for w in waits if w[0] != EMPTY] for waits in turns[3, 4]]
    assert "before its stage is filled" in walk(alone, 3, 4, 2)
    assert walk([[w for w in waits if w[0] != EMPTY] for waits in turns[2, 4]], 2, 4, 2) is None  # (a stage stays with its warp)
