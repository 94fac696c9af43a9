"""The tree replay's two warps stay together (CPU).

m3TreeKernel's text is taken from the source and compiled for the host
with a thread in place of each warp (lane 0 of the walking and of the
staging one), plain stand-ins for the tree, the staging and the scratch,
and a barrier that notices a warp arriving after the other has left the
kernel.  The stand-ins choose the schedules that decide: a world refused
by the step's kernels between the two warps' reads of its status, and a
walk that ends at a malformed tree while the staging warp is late.
"""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "maul3d_b200" / "csrc" / "step.cu"

HARNESS = r"""
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#define __global__
#define __shared__ static
#define __launch_bounds__(n)
#define M3_TREE_THREADS 64
#define M3_TREE_NULL (-1)
#define M3_TREE_TRACKED 1
#define M3_TREE_FULL 2
#define M3GPU_ERR_INVALID 1
#define M3GPU_ERR_CAPACITY 3
struct Dim { uint32_t x; };
static thread_local Dim threadIdx;
static Dim blockIdx = {0};
static int g_scenario;
static int g_lone, g_unstaged;
static bool Stager() { return threadIdx.x >= 32; }
static void Late() { std::this_thread::sleep_for(std::chrono::milliseconds(60)); }

// Two warps; a warp that has left the kernel is never waited for, but an
// arrival after it is counted.
static std::mutex g_lock;
static std::condition_variable g_turn;
static int g_arrived, g_left, g_generation, g_or, g_result;
static int Arrive(int value)
{
    std::unique_lock<std::mutex> hold(g_lock);
    g_or |= value != 0;
    if (g_left > 0)
    {
        g_lone += 1;
        const int alone = g_or;
        g_or = 0;
        return alone;
    }
    if (++g_arrived == 2)
    {
        g_result = g_or;
        g_or = 0;
        g_arrived = 0;
        g_generation += 1;
        g_turn.notify_all();
        return g_result;
    }
    const int generation = g_generation;
    g_turn.wait(hold, [&] { return g_generation != generation || g_left > 0; });
    if (g_generation == generation)
    {
        g_lone += 1;
        g_arrived = 0;
    }
    return g_result;
}
static void Leave()
{
    std::unique_lock<std::mutex> hold(g_lock);
    g_left += 1;
    g_turn.notify_all();
}
#define __syncthreads() Arrive(0)
#define __syncthreads_or(p) Arrive(p)

// A status that one warp already sees and the other not (scenarios 1, 2).
struct Status
{
    int32_t value;
    operator int32_t() const
    {
        return (g_scenario == 1 && Stager()) || (g_scenario == 2 && !Stager()) ? 3 : value;
    }
};
static void atomicExch(Status* s, int32_t v) { s->value = v; }
struct m3WorldScalars
{
    int32_t treeTracked, treeTail, treeRoot, bodyCap, shapeCap, jointCap, pairCap, statusDetail;
    Status status;
    uint64_t phase[16];
};
struct m3WorldView { m3WorldScalars* sc; void* treeNodes; uint8_t* scratch; };
struct m3TreeNode { double a[9]; };
struct m3Scratch { int32_t* treeState; };
static int32_t g_state[33];
static void ScratchCarve(m3Scratch* s, uint8_t*, int, int, int, int, int) { s->treeState = g_state; }
struct m3TreeCursor { int32_t step, move; };
struct Count
{
    int32_t n = 0;
    bool staged = false;
    operator int32_t() const
    {
        if (Stager() && g_scenario == 3)
        {
            Late(); // the walking warp ends its walk meanwhile
        }
        if (!staged)
        {
            g_unstaged += 1;
            return 0;
        }
        return n;
    }
};
struct Box { double lo[6]; };
struct m3TreeChunk { Box box[32]; int32_t shape[32]; int32_t leaf[32]; Count count; int32_t plain; };
static int g_chunks;
static void m3StageTreeChunk(const m3WorldView&, const m3Scratch&, int, int, int, m3TreeCursor*,
                             m3TreeChunk* chunk, int)
{
    for (int k = 0; k < 32; ++k)
    {
        chunk->leaf[k] = chunk->shape[k] = k;
    }
    chunk->count.n = g_chunks++ < 3 ? 32 : 0;
    chunk->count.staged = true;
    chunk->plain = 1;
}
static int g_moved;
struct m3TreeWarp
{
    void* nodes;
    int32_t capacity, root, lane, bound, unbalanced;
    bool tracked;
    bool Move(int32_t, int32_t, const double*)
    {
        return ++g_moved < 40 || g_scenario != 3;
    }
};
@KERNEL@
int main(int argc, char** argv)
{
    g_scenario = argc > 1 ? atoi(argv[1]) : 0;
    static m3WorldScalars sc = {};
    sc.treeTracked = 1;
    m3WorldView view = {&sc, nullptr, nullptr};
    const int32_t order = 0;
    const int32_t steps = 1;
    auto warp = [&](uint32_t first) {
        threadIdx.x = first;
        m3TreeKernel(&view, &order, 1, 32, &steps);
        Leave();
    };
    std::thread walker(warp, 0u);
    std::thread stager(warp, 32u);
    walker.join();
    stager.join();
    printf("%d %d %d %d\n", g_lone, g_unstaged, g_moved, sc.status.value);
    return 0;
}
"""


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    text = SOURCE.read_text()
    kernel = re.search(r"__global__ void __launch_bounds__\(M3_TREE_THREADS\)\s+m3TreeKernel\(.*?\n}\n",
                       text, re.S).group(0)
    kernel = re.sub(r"asm volatile\(.*?\);", "(void)base; (void)piece;", kernel, flags=re.S)
    folder = tmp_path_factory.mktemp("tree")
    (folder / "replay.cpp").write_text(HARNESS.replace("@KERNEL@", kernel))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "replay.cpp", "-o", "replay"],
                   cwd=folder, check=True)

    def run(scenario):
        out = subprocess.run([str(folder / "replay"), str(scenario)], capture_output=True,
                             text=True, timeout=30, check=True).stdout
        return [int(x) for x in out.split()]

    return run


def test_every_chunk_is_replayed(replay):
    assert replay(0) == [0, 0, 96, 0]


@pytest.mark.parametrize("scenario", [1, 2])
def test_a_refusal_between_the_warps_reads(replay, scenario):
    """One decision for the block: both warps replay or both leave, and
    no chunk is read that was not staged."""
    lone, unstaged, moved, _ = replay(scenario)
    assert (lone, unstaged) == (0, 0)
    assert moved in (0, 96)


def test_a_malformed_tree_ends_both_warps_at_the_barrier(replay):
    lone, unstaged, moved, status = replay(3)
    assert (lone, unstaged) == (0, 0)
    assert (moved, status) == (40, 3)
