// Host check of trav_next (lightmetrica-v3_gb300/csrc/lmgpu_dev.cuh) as the eight lanes of a group run
// it: each lane is a thread, and one lane at a time runs, as far as the next barrier of its group, in the
// order given. Whatever the order, all lanes must choose the same node and end at the same stack level,
// as the one-lane form does, and the stack must hold the same words. Prints the number of differences.
#include <algorithm>
#include <condition_variable>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

// One lane at a time: `turn` is the lane that may run. A barrier hands the turn on and returns once all
// eight lanes have come to it.
constexpr int kLanes = 8;
static std::mutex g_m;
static std::condition_variable g_cv;
static int g_order[kLanes], g_turn, g_arrived, g_phase;
static thread_local int t_place;  // the lane's place in the order
struct { unsigned x = 0; } static thread_local threadIdx;
static struct { unsigned x = 1; } blockIdx, gridDim, blockDim;

static void wait_turn(std::unique_lock<std::mutex>& lk) { g_cv.wait(lk, [] { return g_turn == t_place; }); }
static void hand_on() {
    g_turn++;
    g_cv.notify_all();
}
static void __syncwarp(unsigned = 0xffffffffu) {
    std::unique_lock<std::mutex> lk(g_m);
    const int phase = g_phase;
    if (++g_arrived == kLanes) {
        g_arrived = 0;
        g_turn = -1;
        g_phase++;
    }
    hand_on();
    g_cv.wait(lk, [&] { return g_phase != phase; });
    wait_turn(lk);
}

static int __popc(unsigned v) { return __builtin_popcount(v); }
static int __ffs(int v) { return __builtin_ffs(v); }
template <typename T> static T __ldg(const T* p) { return *p; }
// names that other functions of the header use; never called here
static unsigned __ballot_sync(unsigned, bool) { abort(); }
template <typename T> static T __shfl_sync(unsigned, T, int, int = 32) { abort(); }
template <typename T> static T __shfl_xor_sync(unsigned, T, int) { abort(); }
static unsigned __byte_perm(unsigned, unsigned, unsigned) { abort(); }
static unsigned __funnelshift_l(unsigned, unsigned, unsigned) { abort(); }
static unsigned __umulhi(unsigned, unsigned) { abort(); }
static float __uint_as_float(unsigned) { abort(); }
static unsigned __float_as_uint(float) { abort(); }
static float __fmul_rn(float, float) { abort(); }
static float __fadd_rn(float, float) { abort(); }
static float __fsub_rn(float, float) { abort(); }
static float __fdiv_rn(float, float) { abort(); }
static float __fsqrt_rn(float) { abort(); }
static int atomicAdd(int*, int) { abort(); }
static void __syncthreads() { abort(); }
template <typename T> static T min(T a, T b) { return a < b ? a : b; }
template <typename T> static T max(T a, T b) { return a > b ? a : b; }
using std::signbit;

#include "lmgpu_dev.cuh"

using namespace lmgpu;

struct Step {
    uint32_t base, imask, inner;
};

int main(int argc, char** argv) {
    std::mt19937 rng(argc > 1 ? unsigned(atoi(argv[1])) : 1u);
    const int depth = 12, rounds = 200;
    int bad = 0, pops_left = 0;
    for (int r = 0; r < rounds; r++) {
        // the nodes a ray meets: inner children entered (often none, so that entries are popped)
        std::vector<Step> steps(24);
        for (Step& s : steps) {
            s.base = rng() % 100000u;
            s.imask = rng() & 0xffu;
            s.inner = rng() % 2u ? 0u : s.imask & rng();
        }
        const uint32_t oct = rng() % 8u;
        Bvh8 bvh{};
        bvh.depth = depth;
        // the one-lane form
        std::vector<uint2> ref_stk(depth);
        std::vector<std::pair<uint32_t, int>> ref;
        Trav s0{};
        s0.oct = oct;
        s0.inst_sp = -1;
        for (const Step& st : steps) {
            if (!trav_next<false>(bvh, s0, st.base, st.imask, st.inner, ref_stk.data(), 1)) break;
            ref.emplace_back(s0.node, s0.sp);
            if (s0.node == kNoNode) break;
            pops_left += st.inner == 0u;
        }
        // the group, in an order of its own
        for (int i = 0; i < kLanes; i++) g_order[i] = i;
        if (r >= rounds / 2) std::shuffle(g_order, g_order + kLanes, rng);
        g_turn = 0;
        g_arrived = g_phase = 0;
        std::vector<uint2> stk(depth);
        std::vector<std::pair<uint32_t, int>> got[kLanes];
        std::vector<std::thread> lanes;
        for (int i = 0; i < kLanes; i++)
            lanes.emplace_back([&, i] {
                t_place = i;
                threadIdx.x = unsigned(g_order[i]);
                {
                    std::unique_lock<std::mutex> lk(g_m);
                    wait_turn(lk);
                }
                Trav s{};
                s.oct = oct;
                s.inst_sp = -1;
                for (size_t k = 0; k < ref.size(); k++) {
                    trav_next<false, true>(bvh, s, steps[k].base, steps[k].imask, steps[k].inner, stk.data(), 1);
                    got[i].emplace_back(s.node, s.sp);
                    // a lane that has left its group's path would wait for barriers the others never reach
                    if (got[i].back() != ref[k]) {
                        fprintf(stderr, "lane %d of order place %d differs at step %zu\n", g_order[i], i, k);
                        printf("differences 1\n");
                        fflush(stdout);
                        _Exit(1);
                    }
                    __syncwarp();  // the next step of the loop
                }
                std::unique_lock<std::mutex> lk(g_m);
                hand_on();
            });
        for (auto& t : lanes) t.join();
        for (int i = 0; i < kLanes; i++) bad += got[i] != ref;
        for (int i = 0; i < s0.sp; i++) bad += stk[i].x != ref_stk[i].x || stk[i].y != ref_stk[i].y;
    }
    printf("differences %d pops %d\n", bad, pops_left);
    return bad != 0 || pops_left < rounds;
}
