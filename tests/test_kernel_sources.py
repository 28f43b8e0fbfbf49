"""Rules that the kernels' sources have to keep and that no run can show to hold: read here as text, without a GPU."""
import glob
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nvfp4_cutlass_b200", "csrc")
KERNELS = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")))


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def enclosing(text, at):
    """Headers of the blocks around position `at`, and the names of the calls whose argument lists are open there."""
    blocks, calls, header = [], [], 0
    for i, c in enumerate(text[:at]):
        if c == "{":
            blocks.append(text[header:i])
            header = i + 1
        elif c == "}":
            blocks.pop()
            header = i + 1
        elif c == ";":
            header = i + 1
        elif c == "(":
            calls.append(re.search(r"[\w:]*$", text[:i]).group(0))
        elif c == ")":
            calls.pop()
    return blocks, calls


@pytest.mark.parametrize("name", KERNELS)
def test_a_warp_waits_as_one(name):
    """A bounded wait is made by one thread, or the warp votes on its outcome: lanes that leave a poll at different times
    must not reach a warp-wide instruction apart, and none may give up alone."""
    text = source(name)
    for m in re.finditer(r"ptx::mbar_wait\w*", text):
        blocks, calls = enclosing(text, m.start())
        by_one = any(re.search(r"\b(lane|threadIdx\.x) == 0\b", b) for b in blocks) or \
            "threadIdx.x == 0 &&" in text[text.rfind(";", 0, m.start()):m.start()]
        assert by_one or "ptx::all_lanes" in calls, f"{name}:{text.count(chr(10), 0, m.start()) + 1}"


def test_warp_wide_instructions_start_converged():
    """Allocation, release and the cluster barrier follow roles that one lane runs alone."""
    text = source("ptx.cuh")
    for mnemonic in ("tcgen05.alloc", "tcgen05.dealloc", "barrier.cluster.arrive"):
        places = [m.start() for m in re.finditer(re.escape(mnemonic), text)]
        assert places
        for at in places:
            assert "__syncwarp();" in text[text.rfind("{", 0, text.rfind("asm", 0, at)):at], mnemonic


RING_CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include "ring.cuh"
using nvfp4::gemm::Ring;
using nvfp4::gemm::drain_ring;

// `blocks` K blocks through the ring: the producer waits for a group's last use before it opens it again, the tensor core
// commits every group that is full.  Parity p of a barrier that has been opened u times stands for use u - 1 when
// p == (u - 1) % 2; a barrier that was never opened passes for parity 1.
template <uint32_t kDepth, uint32_t kGroup> bool check(uint32_t blocks)
{
    constexpr uint32_t kGroups = kDepth / kGroup;
    uint32_t committed[kGroups] = {}, awaited[kGroups] = {};
    for (uint32_t b = 0; b < blocks; ++b)
        if (b % kGroup == kGroup - 1) ++committed[b / kGroup % kGroups];
    Ring r;
    // what the producer has waited for by the time of its last load: use u of a group before it opens use u + 1
    uint32_t opened[kGroups] = {};
    for (uint32_t b = 0; b < blocks; ++b) {
        if (r.slot % kGroup == 0) awaited[r.slot / kGroup] = opened[r.slot / kGroup]++;
        r.template advance<kDepth>();
    }
    bool fine = true;
    drain_ring<kDepth, kGroup>(r, [&](uint32_t group, uint32_t parity) {
        // the parity names the last use that was opened: it has to be one that will be committed
        if (opened[group] == 0) { fine = fine && parity == 1; return true; }
        fine = fine && ((opened[group] - 1) & 1u) == parity && committed[group] == opened[group];
        awaited[group] = opened[group];
        return true;
    });
    for (uint32_t g = 0; g < kGroups; ++g) fine = fine && awaited[g] == committed[g];
    return fine;
}
template <uint32_t kDepth, uint32_t kGroup> void all()
{
    for (uint32_t blocks = 0; blocks <= 4 * kDepth + 3; ++blocks)
        if (!check<kDepth, kGroup>(blocks)) { std::printf("depth %u group %u blocks %u\n", kDepth, kGroup, blocks); std::exit(1); }
}
int main()
{
    all<2, 1>(); all<3, 1>(); all<4, 1>(); all<5, 1>(); all<7, 1>(); all<10, 1>(); all<12, 1>();
    all<4, 2>(); all<6, 2>(); all<8, 2>(); all<6, 3>(); all<12, 4>();
    return 0;
}
"""


def test_the_drain_awaits_every_commit_and_no_other(tmp_path):
    program = tmp_path / "ring.cpp"
    program.write_text(RING_CHECK)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, str(program), "-o", str(tmp_path / "ring")], check=True)
    assert subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True).stdout == ""


@pytest.mark.parametrize("name", [k for k in KERNELS if "tcgen05_commit" in source(k) and k.startswith("gemm_")])
def test_every_ring_freed_by_commits_is_drained(name):
    """No block leaves before the commits to its ring barriers have arrived: each barrier array that a commit signals, the
    accumulator's apart (the epilogue waits for all of those), has a drain in its kernel."""
    text = source(name)
    for kernel in text.split("__global__")[1:]:
        signalled = set(re.findall(r"tcgen05_commit\w*\((\w+)", kernel)) - {"tmem_full"}
        drained = set(re.findall(r"drain_ring<.*?mbar_wait[\w<>]*\((\w+)", kernel, re.S))
        assert signalled <= drained, (name, signalled, drained)


TURN_CHECK = r"""
#include <cstdint>
#include <cstdio>
#include <random>
#include "ring.cuh"
using nvfp4::gemm::wait_turn;

// One CTA of the fused cluster kernel as a model: the producer loads blocks in order, loads land in any order, kGroups groups
// take blocks in turn, the tensor core takes them in order.  Roles step in a random order, a role that waits stays where it is.
// `uses` counts a barrier's completed uses; a wait sees their parity only.  Returns false when a wait passed too early.
template <uint32_t kDepth, uint32_t kGroups, uint32_t kBlocks> bool run(std::mt19937& rng)
{
    uint32_t a_full[kDepth] = {}, a_empty[kDepth] = {}, share_full[kDepth] = {}, p_empty[kDepth] = {};
    bool landed[kBlocks] = {}, issued[kBlocks] = {};
    uint32_t next_load = 0, next_mma = 0, at[kGroups], stage[kGroups] = {};
    bool early = false;
    auto passes = [&](uint32_t uses, uint32_t parity) { return ((uses - 1u) & 1u) == parity; };
    for (uint32_t g = 0; g < kGroups; ++g) at[g] = g;
    for (uint32_t steps = 0; steps < 400000 && next_mma < kBlocks; ++steps) {
        const uint32_t who = rng() % (kGroups + 3);
        if (who < kGroups) {
            const uint32_t it = at[who], slot = it % kDepth, use = it / kDepth;
            if (it >= kBlocks) continue;
            if (stage[who] == 0) {                               // wait for the tile, then hand its slot back
                if (!wait_turn<kDepth, kGroups>(it, [&](uint32_t i, uint32_t p) { return passes(share_full[i], p); },
                                                [&](uint32_t i, uint32_t p) { return passes(a_full[i], p); })) continue;
                if (a_full[slot] != use + 1) early = true;
                ++a_empty[slot];
                stage[who] = 1;
            } else {                                             // wait for the slot of the products, then write them
                if (!passes(p_empty[slot], (use & 1u) ^ 1u)) continue;
                if (p_empty[slot] != use) early = true;
                ++share_full[slot];
                stage[who] = 0;
                at[who] += kGroups;
            }
        } else if (who == kGroups) {                             // producer
            if (next_load < kBlocks && a_empty[next_load % kDepth] == next_load / kDepth) issued[next_load++] = true;
        } else if (who == kGroups + 1) {                         // some load lands
            const uint32_t b = next_load == 0 ? 0 : next_load - 1 - rng() % (next_load < kDepth ? next_load : kDepth);
            if (issued[b] && !landed[b] && rng() % 8 == 0) { landed[b] = true; ++a_full[b % kDepth]; }
        } else if (share_full[next_mma % kDepth] == next_mma / kDepth + 1) {
            ++p_empty[next_mma % kDepth];
            ++next_mma;
        }
        if (early) return false;
    }
    return next_mma == kBlocks;
}
int main()
{
    std::mt19937 rng(1);
    for (int i = 0; i < 3000; ++i)
        if (!run<5, 3, 64>(rng) || !run<4, 1, 64>(rng) || !run<3, 2, 48>(rng) || !run<5, 4, 64>(rng)) { std::printf("run %d\n", i); return 1; }
    return 0;
}
"""


def test_groups_in_turn_never_pass_a_wait_early(tmp_path):
    program = tmp_path / "turn.cpp"
    program.write_text(TURN_CHECK)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(program), "-o", str(tmp_path / "turn")], check=True)
    assert subprocess.run([str(tmp_path / "turn")], capture_output=True, text=True).stdout == ""
    text = source("gemm_cluster.cu")                                   # the only kernel whose roles take blocks in turn
    assert re.search(r"wait_turn<C::kDepthA, C::kGroups>\(\s*it,.*?share_full \+ i,.*?a_full \+ i,", text, re.S)
    assert not any("% C::kGroups" in source(k) for k in KERNELS if k != "gemm_cluster.cu")


def handed_back_too_early(text):
    """Places where a slot that a bulk or TMA load fills goes back to its producer while plain loads of it may still be under way:
    since the last load (transform_tile's among them) there is neither a proxy fence nor anything that used what was loaded (scales
    stored to tensor memory, an output row stored)."""
    bad = []
    for m in re.finditer(r"ptx::mbar_arrive\((?:a_empty|sf_free|empty) \+", text):
        load = max(text.rfind("ptx::lds", 0, m.start()), text.rfind("transform_tile<", 0, m.start()))
        if not re.search(r"fence_proxy_async_smem\(\)|tmem_st_wait\(\)|\by\[[^;]*\] = make_uint4", text[load:m.start()]):
            bad.append(text.count(chr(10), 0, m.start()) + 1)
    return bad


@pytest.mark.parametrize("name", KERNELS)
def test_loads_of_a_slot_end_before_it_is_handed_back(name):
    """A plain load is ordered before the asynchronous write that refills its slot by a proxy fence between the load and the arrive
    that lets the producer go on.  Without it rows of the next tile turned up in 7 to 11 of 40 decode calls (120 experts, N = 1280,
    K = 3456)."""
    assert handed_back_too_early(source(name)) == []


def test_the_rule_on_handed_back_slots_sees_a_missing_fence():
    fence = re.compile(r"ptx::fence_proxy_async_smem\(\);(?=\s*__syncwarp\(\);\s*if \(lane == 0\) \{?\s*ptx::mbar_arrive\(a_empty)")
    for name in ("gemm_cluster.cu", "gemm_normal.cu", "gemm_swap.cu"):
        text = source(name)
        assert len(fence.findall(text)) == 1 and len(handed_back_too_early(fence.sub("", text))) == 1
    # the decode kernel hands a slot back in two places, of which a form has one; the later one lies behind both fences
    late = re.compile(r"ptx::fence_proxy_async_smem\(\);(?=\s*__syncwarp\(\);\s*if \(lane == 0\) \{\s*if constexpr \(!kGeneral\) ptx::mbar_arrive\(a_empty)")
    text = source("gemm_swap.cu")
    assert len(late.findall(text)) == 1 and len(handed_back_too_early(fence.sub("", late.sub("", text)))) == 2
    for name, used in (("gemm_split.cu", "ptx::tmem_st_wait();"), ("moe_glue.cu", "y[t * y_ld16 + c] = make_uint4(ow[0], ow[1], ow[2], ow[3]);")):
        assert used in source(name) and handed_back_too_early(source(name).replace(used, ""))
    places = sum(len(re.findall(r"ptx::mbar_arrive\((?:a_empty|sf_free|empty) \+", source(k))) for k in KERNELS)
    assert places == 6                                     # decode x 2, fused x 2, pair, bulk combine
