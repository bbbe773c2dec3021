// GPU build of the 8-wide quantized BVH (the node and triangle layout of bvh_build.h), the device
// counterpart of build_bvh8:
//
//   1. triangle boxes and centroid bounds; 30-bit Morton codes of the centroids;
//   2. a radix sort of (code, triangle) pairs (CUB);
//   3. PLOC clustering (Meister & Bittner, "Parallel Locally-Ordered Clustering for Bounding
//      Volume Hierarchy Construction", TVCG 2018): every cluster finds the neighbour within
//      kRadius places of the sorted order whose merged box has the smallest surface area; mutual
//      nearest neighbours merge into a new binary node; compaction by prefix sums; repeat until
//      one cluster is left. Node ids come from the prefix sums, so the tree is deterministic;
//   4. the SAH-optimal 8-wide collapse cost of every binary node (Ylitie, Karras & Laine, HPG
//      2017; the same recurrence and constants as the host builder), computed when the node is
//      created, since its children are final by then;
//   5. top-down emission, one launch per level: each wide node gathers its children from the
//      collapse decisions, orders them by octant, takes contiguous slots for its internal children
//      and its leaf triangles (atomics), writes the triangle records (p1, e1 = p2 - p1, e2 = p3 - p1
//      rounded once in fp32, as Tri's constructor) and quantizes the child boxes exactly as the
//      host builder does (outward rounding plus one quantum of margin, checked in double: the
//      planes p + q * 2^e are exact in double for the exponents chosen).
//
// The reference builds its binary SAH tree with full sorts on the host (accel_sahbvh.cpp:127-267).
// Closest hits do not depend on the tree (the traversal's tie rule is the smaller triangle index),
// so any of these builders gives the same hits.
#include <cub/device/device_radix_sort.cuh>

#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "bvh_build.h"
#include "runtime.h"

namespace lmgpu {
namespace gpubuild {

constexpr int kMaxLeaf = 3;      // triangles per leaf child (3 bits of meta hold the count)
// PLOC neighbourhood: kRadius clusters on either side. Trace speed of the resulting trees on
// the 3.8M-triangle headline scene (64 spp, Mrays/s; the host SAH builder's tree: 2,680):
// radius 4 -> 2,594, 6 -> 2,684, 8 -> 2,636, 16 -> 2,497, 32 -> 2,540. On random-triangle soups of
// 1.5k-160k triangles every radius from 4 to 8 stays within 1-7 % of the host builder's trees.
constexpr int kRadius = 6;
constexpr int kBlock = 256;
constexpr float kCNode = 1.0f, kCPrim = 0.3f;

// error bits
constexpr int kErrNonFinite = 1, kErrQuantize = 2, kErrLayout = 4;

struct Nodes {
    float4* lo;       // binary node boxes (w unused)
    float4* hi;
    int32_t* left;    // -1 for a leaf
    int32_t* right;   // leaf: its triangle
    int32_t* count;   // triangles below
    float* cost;      // 8 per node: collapse cost with at most i slots of the parent
    int8_t* dec;      // 8 per node: i = 1: 0 leaf / 1 wide node; i > 1: 0 = as i - 1, k = split k | i - k
    int8_t* dnode;    // the node's own split of 8 slots between its children
};

__device__ inline float box_area(float4 lo, float4 hi) {
    if (!(hi.x >= lo.x)) return 0.f;
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return 2.f * (dx * dy + dy * dz + dz * dx);
}

// float -> uint32 with the same order (atomicMin / atomicMax on floats)
__device__ inline uint32_t ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float unordered(uint32_t u) {
    const uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    float f;
    memcpy(&f, &b, 4);
    return f;
}

// Triangle boxes, centroids, centroid bounds (cb: 3 ordered minima then 3 ordered maxima).
__global__ void k_prep(const float* __restrict__ P, int64_t n, float4* __restrict__ tlo, float4* __restrict__ thi,
                       float4* __restrict__ cen, uint32_t* cb, int* err) {
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        float v[9];
        bool finite = true;
        for (int k = 0; k < 9; k++) {
            v[k] = P[9 * i + k];
            finite = finite && isfinite(v[k]);
        }
        if (!finite) atomicOr(err, kErrNonFinite);
        float lo[3], hi[3], c[3];
        for (int a = 0; a < 3; a++) {
            lo[a] = fminf(fminf(v[a], v[3 + a]), v[6 + a]);
            hi[a] = fmaxf(fmaxf(v[a], v[3 + a]), v[6 + a]);
            if (!isfinite(lo[a]) || !isfinite(hi[a])) lo[a] = hi[a] = 0.f;
            c[a] = 0.5f * (lo[a] + hi[a]);
            mn[a] = fminf(mn[a], c[a]);
            mx[a] = fmaxf(mx[a], c[a]);
        }
        tlo[i] = make_float4(lo[0], lo[1], lo[2], 0.f);
        thi[i] = make_float4(hi[0], hi[1], hi[2], 0.f);
        cen[i] = make_float4(c[0], c[1], c[2], 0.f);
    }
    for (int a = 0; a < 3; a++) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
    }
    if ((threadIdx.x & 31) == 0 && mn[0] <= mx[0]) {
        for (int a = 0; a < 3; a++) {
            atomicMin(cb + a, ordered(mn[a]));
            atomicMax(cb + 3 + a, ordered(mx[a]));
        }
    }
}

__device__ inline uint32_t spread10(uint32_t x) {  // 10 bits -> every third bit
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

__global__ void k_morton(const float4* __restrict__ cen, int64_t n, const uint32_t* __restrict__ cb,
                         uint32_t* __restrict__ keys, int32_t* __restrict__ vals) {
    float lo[3], inv[3];
    for (int a = 0; a < 3; a++) {
        lo[a] = unordered(cb[a]);
        const float ext = unordered(cb[3 + a]) - lo[a];
        inv[a] = ext > 0.f ? 1024.f / ext : 0.f;
    }
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const float4 c = cen[i];
        const float cc[3] = {c.x, c.y, c.z};
        uint32_t q[3];
        for (int a = 0; a < 3; a++) q[a] = uint32_t(fminf(fmaxf((cc[a] - lo[a]) * inv[a], 0.f), 1023.f));
        keys[i] = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
        vals[i] = int32_t(i);
    }
}

// Collapse cost of node `id` from its children's (their costs are final).
__device__ void collapse_cost(const Nodes& N, int32_t id, int32_t l, int32_t r, float4 lo, float4 hi, int32_t count,
                              int W) {
    const float A = box_area(lo, hi);
    const float cleaf = count <= kMaxLeaf ? A * kCPrim * float(count) : INFINITY;
    float* c = N.cost + size_t(id) * 8;
    int8_t* d = N.dec + size_t(id) * 8;
    if (l < 0) {
        for (int i = 0; i < 8; i++) { c[i] = cleaf; d[i] = 0; }
        N.dnode[id] = 1;
        return;
    }
    float cl[8], cr[8];
    for (int i = 0; i < 8; i++) { cl[i] = N.cost[size_t(l) * 8 + i]; cr[i] = N.cost[size_t(r) * 8 + i]; }
    float dist[9];
    int8_t dk[9];
    for (int j = 2; j <= 8; j++) {
        dist[j] = INFINITY;
        dk[j] = 1;
        for (int k = 1; k < j; k++) {
            const float v = cl[k - 1] + cr[j - k - 1];
            if (v < dist[j]) { dist[j] = v; dk[j] = int8_t(k); }
        }
    }
    const float cnode = A * kCNode + dist[W];
    float c0 = fminf(cleaf, cnode);
    c[0] = c0;
    d[0] = cleaf <= cnode ? 0 : 1;
    N.dnode[id] = dk[W];
    float prev = c0;
    for (int i = 2; i <= 8; i++) {
        if (prev <= dist[i]) { c[i - 1] = prev; d[i - 1] = 0; }
        else { c[i - 1] = dist[i]; d[i - 1] = dk[i]; prev = dist[i]; }
    }
}

// Clusters left and the next binary node's id, kept on the device so that several passes run between
// two reads by the host. Pass i reads state[i & 1] and leaves state[1 - (i & 1)].
struct PlocState {
    int32_t m, next_id;
};

// Leaves in Morton order: leaf k holds triangle vals[k]; every leaf starts as its own cluster.
__global__ void k_leaves(const int32_t* __restrict__ vals, int64_t n, const float4* __restrict__ tlo,
                         const float4* __restrict__ thi, Nodes N, int32_t* __restrict__ clusters, PlocState* state) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *state = PlocState{int32_t(n), int32_t(n)};
    for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x) {
        const int32_t t = vals[k];
        const float4 lo = tlo[t], hi = thi[t];
        N.lo[k] = lo;
        N.hi[k] = hi;
        N.left[k] = -1;
        N.right[k] = t;
        N.count[k] = 1;
        collapse_cost(N, int32_t(k), -1, -1, lo, hi, 1, 8);
        clusters[k] = int32_t(k);
    }
}

__device__ inline float4 box_min(float4 a, float4 b) { return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.f); }
__device__ inline float4 box_max(float4 a, float4 b) { return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.f); }

// Area of the merged box, then the position: the order in which neighbours are preferred.
__device__ inline unsigned long long merged_key(float4 alo, float4 ahi, float4 blo, float4 bhi, int32_t j) {
    const float area = box_area(box_min(alo, blo), box_max(ahi, bhi));
    return (static_cast<unsigned long long>(__float_as_uint(area)) << 32) | uint32_t(j);
}

// Exclusive prefix sum over the block's threads of (a, b) pairs packed as a << 32 | b; *total is the
// block's sum. `shared`: one word per warp. Called by all threads of the block.
__device__ inline unsigned long long block_scan(unsigned long long v, unsigned long long* shared, unsigned long long* total) {
    const int lane = int(threadIdx.x & 31u), warp = int(threadIdx.x >> 5), warps = int(blockDim.x >> 5);
    unsigned long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) shared[warp] = inc;
    __syncthreads();
    unsigned long long before = 0, all = 0;
    for (int w = 0; w < warps; w++) {
        const unsigned long long u = shared[w];
        before += w < warp ? u : 0ull;
        all += u;
    }
    *total = all;
    return before + inc - v;
}

// What position i does, given its nearest neighbour j and j's: a << 32 | b with a = 1 if i starts a
// merge (a mutual pair, i the smaller position) and b = 1 if i stays a cluster (no merge, or the
// merge's first position).
__device__ inline unsigned long long merge_flags(int32_t i, int32_t j, int32_t nn_j) {
    const bool mutual = j != i && nn_j == i, lead = mutual && i < j;
    return (static_cast<unsigned long long>(lead) << 32) | ((!mutual || lead) ? 1ull : 0ull);
}

// Nearest neighbour of every cluster within kRadius places: the smallest merged surface area, ties
// to the smaller position (a total order, so the closest pair is always mutual), and the block's
// sums of merge_flags. Boxes and neighbours of the block's window are staged in shared memory; the
// neighbours of kRadius places on either side are found a second time here rather than in a launch
// of their own (a pass was five launches: neighbours, flags, a two-kernel scan and the merge).
__global__ void __launch_bounds__(kBlock) k_nearest(const int32_t* __restrict__ clusters, const PlocState* __restrict__ state,
                                                    const float4* __restrict__ nlo, const float4* __restrict__ nhi,
                                                    int32_t* __restrict__ nn, unsigned long long* __restrict__ sums) {
    constexpr int kHalo = 2 * kRadius, kNear = kBlock + 2 * kRadius;
    __shared__ float4 slo[kBlock + 2 * kHalo], shi[kBlock + 2 * kHalo];
    __shared__ int32_t snn[kNear];
    __shared__ unsigned long long warp_sum[kBlock / 32];
    const int32_t m = state->m, first = int32_t(blockIdx.x) * kBlock;
    if (first >= m) {
        if (threadIdx.x == 0) sums[blockIdx.x] = 0ull;
        return;
    }
    for (int k = threadIdx.x; k < kBlock + 2 * kHalo; k += kBlock) {
        const int32_t p = first - kHalo + k;
        if (p >= 0 && p < m) {
            const int32_t c = clusters[p];
            slo[k] = nlo[c];
            shi[k] = nhi[c];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kNear; k += kBlock) {
        const int32_t i = first - kRadius + k;
        if (i < 0 || i >= m) continue;
        const float4 alo = slo[k + kRadius], ahi = shi[k + kRadius];
        unsigned long long best = ~0ull;
        for (int32_t j = max(0, i - kRadius); j <= min(m - 1, i + kRadius); j++) {
            if (j == i) continue;
            const unsigned long long key = merged_key(alo, ahi, slo[j - first + kHalo], shi[j - first + kHalo], j);
            best = key < best ? key : best;
        }
        snn[k] = m > 1 ? int32_t(best & 0xffffffffu) : i;
    }
    __syncthreads();
    const int32_t i = first + int32_t(threadIdx.x);
    unsigned long long f = 0ull, total;
    if (i < m) {
        const int32_t j = snn[threadIdx.x + kRadius];
        nn[i] = j;
        f = merge_flags(i, j, snn[j - first + kRadius]);
    }
    block_scan(f, warp_sum, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Prefix sums of the blocks' sums, in place, and the state after the pass.
__global__ void __launch_bounds__(1024) k_scan_blocks(unsigned long long* sums, int32_t blocks, const PlocState* __restrict__ state,
                                                      PlocState* next) {
    __shared__ unsigned long long warp_sum[32];
    unsigned long long run = 0;
    for (int32_t base = 0; base < blocks; base += 1024) {
        const int32_t k = base + int32_t(threadIdx.x);
        unsigned long long total;
        const unsigned long long v = k < blocks ? sums[k] : 0ull, ex = block_scan(v, warp_sum, &total);
        if (k < blocks) sums[k] = run + ex;
        run += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *next = PlocState{int32_t(run & 0xffffffffu), state->next_id + int32_t(run >> 32)};
}

// The merge of clusters a and b as binary node `id` with box (lo, hi).
__device__ inline void merge_node(const Nodes& N, int32_t id, int32_t a, int32_t b, float4 lo, float4 hi, int W) {
    const int32_t cnt = N.count[a] + N.count[b];
    N.lo[id] = lo;
    N.hi[id] = hi;
    N.left[id] = a;
    N.right[id] = b;
    N.count[id] = cnt;
    collapse_cost(N, id, a, b, lo, hi, cnt, W);
}
__global__ void __launch_bounds__(kBlock) k_merge(const int32_t* __restrict__ cin, const PlocState* __restrict__ state,
                                                  const int32_t* __restrict__ nn, const unsigned long long* __restrict__ before,
                                                  Nodes N, int32_t* __restrict__ cout, int W) {
    __shared__ unsigned long long warp_sum[kBlock / 32];
    const int32_t i = int32_t(blockIdx.x) * kBlock + int32_t(threadIdx.x), m = state->m;
    if (int32_t(blockIdx.x) * kBlock >= m) return;
    const int32_t j = i < m ? nn[i] : i;
    const unsigned long long f = i < m ? merge_flags(i, j, nn[j]) : 0ull;
    unsigned long long total;
    const unsigned long long s = before[blockIdx.x] + block_scan(f, warp_sum, &total);
    if (!(f & 1ull)) return;
    const int32_t slot = int32_t(s & 0xffffffffu);
    if (f >> 32) {
        const int32_t id = state->next_id + int32_t(s >> 32);
        const int32_t a = cin[i], b = cin[j];
        merge_node(N, id, a, b, box_min(N.lo[a], N.lo[b]), box_max(N.hi[a], N.hi[b]), W);
        cout[slot] = id;
    } else {
        cout[slot] = cin[i];
    }
}

// The root and what the host reports about it.
struct RootInfo {
    int32_t root;
    float cost;
    float lo[3], hi[3];
};

// The last kLast clusters: every remaining pass in one block, positions and boxes in shared memory,
// the same merges and node ids as the passes above. A pass shrinks the list by about a quarter, so
// more than half of a build's passes have fewer clusters than one block has threads; as five
// launches and a read by the host each they took 40 us, here about 4.
constexpr int kLast = 1024;
__global__ void __launch_bounds__(kLast) k_last_passes(const int32_t* __restrict__ clusters, const PlocState* __restrict__ state,
                                                       Nodes N, int W, RootInfo* out, int* err) {
    __shared__ float4 slo[kLast], shi[kLast];
    __shared__ int32_t sid[kLast], snn[kLast];
    __shared__ unsigned long long warp_sum[32];
    const int i = int(threadIdx.x);
    int m = state->m, next_id = state->next_id;
    if (i < m) {
        const int32_t c = clusters[i];
        sid[i] = c;
        slo[i] = N.lo[c];
        shi[i] = N.hi[c];
    }
    __syncthreads();
    while (m > 1) {
        if (i < m) {
            unsigned long long best = ~0ull;
            const float4 alo = slo[i], ahi = shi[i];
            for (int j = max(0, i - kRadius); j <= min(m - 1, i + kRadius); j++) {
                if (j == i) continue;
                const unsigned long long key = merged_key(alo, ahi, slo[j], shi[j], j);
                best = key < best ? key : best;
            }
            snn[i] = int32_t(best & 0xffffffffu);
        }
        __syncthreads();
        const int j = i < m ? snn[i] : i;
        const unsigned long long f = i < m ? merge_flags(i, j, snn[j]) : 0ull;
        const bool keep = f & 1ull, lead = f >> 32;
        unsigned long long total;
        const unsigned long long ex = block_scan(f, warp_sum, &total);
        int32_t id = 0;
        float4 lo, hi;
        if (keep) {
            id = sid[i];
            lo = slo[i];
            hi = shi[i];
            if (lead) {
                const int32_t a = id, b = sid[j];
                id = next_id + int32_t(ex >> 32);
                lo = box_min(lo, slo[j]);
                hi = box_max(hi, shi[j]);
                merge_node(N, id, a, b, lo, hi, W);
            }
        }
        const int merges = int(total >> 32), left = int(total & 0xffffffffu);
        if (merges < 1 || left != m - merges) {  // the same in all threads
            if (i == 0) atomicOr(err, kErrLayout);
            break;
        }
        __syncthreads();
        if (keep) {
            const int slot = int(ex & 0xffffffffu);
            sid[slot] = id;
            slo[slot] = lo;
            shi[slot] = hi;
        }
        m = left;
        next_id += merges;
        __syncthreads();
    }
    if (i == 0) {
        const int32_t r = sid[0];
        const float4 lo = slo[0], hi = shi[0];
        *out = RootInfo{r, N.cost[size_t(r) * 8], {lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
    }
}

// ---- emission ------------------------------------------------------------------------------

// Counters of the emission, one host read for all of them. `now` is copied to the ring after every
// level, so that the error word a level reads is the same in all of its threads.
struct LevelEnd {
    int32_t wide_count;
    int err;
};
struct EmitState {
    LevelEnd now;
    int32_t tri_count;
    LevelEnd level[8];  // ring: level l holds the wide nodes [level[l & 7], level[(l + 1) & 7])
};

struct Emit {
    Nodes N;
    const float* P;          // input triangles (p1, p2, p3)
    uint32_t* nodes;         // 20 words per wide node
    float4* tris;            // 3 float4 per triangle record
    int32_t* tri_slot;       // flattened triangle index -> record
    int32_t* q_bin;          // wide node -> its binary node
    EmitState* st;
    const RootInfo* root;
    int32_t wide_cap;
    int width;               // children per node (2..8)
};

__device__ inline uint32_t fbits(float f) { return __float_as_uint(f); }

// smallest biased exponent eb with 2^(eb-127) >= v (bvh_build.cpp exponent_for)
__device__ int exponent_for(double v) {
    if (!(v > 0)) return 1;
    int e2;
    const double mm = frexp(v, &e2);
    int eb = (mm == 0.5 ? e2 - 1 : e2) + 127;
    return min(254, max(1, eb));
}

// Eight lanes per wide node, lane s for child slot s. One thread per node ran the slot assignment and
// the quantization (both in double, as on the host, and double is slow here) for its eight children
// in turn: 250 us per level of a 200k-triangle build however few nodes it had, 55 us now.
constexpr int kEmitBlock = 128;
__global__ void __launch_bounds__(kEmitBlock) k_emit(Emit E, int level) {
    const Nodes& N = E.N;
    const int lane = int(threadIdx.x & 31u), s = lane & 7;
    const unsigned gm = 0xffu << (lane & 24);
    const LevelEnd end = E.st->level[(level + 1) & 7];
    // a node with an error has counted its children and not written them, and the host looks only after
    // four levels (merged boxes whose area overflows get here)
    if (end.err) return;
    const int32_t w1 = end.wide_count, root = E.root->root;
    auto from = [&](auto v, int src) { return __shfl_sync(gm, v, src, 8); };
    for (int32_t w = E.st->level[level & 7].wide_count + (int32_t(blockIdx.x) * kEmitBlock + int32_t(threadIdx.x)) / 8; w < w1;
         w += int32_t(gridDim.x) * (kEmitBlock / 8)) {
        const int32_t bin = E.q_bin[w];
        // the node's children (binary node ids), depth-first left before right: child i goes to lane i
        int32_t ch = -1;
        bool leaf = false;
        int nch = 0;
        bool bad = false;
        if (N.left[bin] < 0 || (bin == root && N.dec[size_t(bin) * 8] == 0)) {
            if (s == 0) {
                ch = bin;
                leaf = true;
            }
            nch = 1;
        } else {
            int32_t sm[16];
            int si[16];
            int sp = 0;
            const int k0 = N.dnode[bin];
            sm[sp] = N.right[bin]; si[sp++] = E.width - k0;
            sm[sp] = N.left[bin]; si[sp++] = k0;
            while (sp > 0 && !bad) {
                const int32_t m = sm[--sp];
                int i = si[sp];
                while (i > 1 && N.dec[size_t(m) * 8 + i - 1] == 0) i--;
                if (i == 1) {
                    if (nch >= 8) { bad = true; break; }
                    if (nch == s) {
                        ch = m;
                        leaf = N.left[m] < 0 || N.dec[size_t(m) * 8] == 0;
                    }
                    nch++;
                    continue;
                }
                const int k = N.dec[size_t(m) * 8 + i - 1];
                if (sp + 2 > 16) { bad = true; break; }
                sm[sp] = N.right[m]; si[sp++] = i - k;
                sm[sp] = N.left[m]; si[sp++] = k;
            }
        }
        if (bad) {  // the same in all lanes of the group
            atomicOr(&E.st->now.err, kErrLayout);
            continue;
        }
        // octant-ordered slots (bvh_build.cpp: greedy on dot(centroid - center, octant direction))
        float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
        int cnt = 0;
        if (ch >= 0) {
            lo = N.lo[ch];
            hi = N.hi[ch];
            cnt = N.count[ch];
        }
        float4 nlo = lo, nhi = hi;
        for (int o = 1; o < 8; o <<= 1) {
            auto other = [&](float v) { return __shfl_xor_sync(gm, v, o); };
            nlo = box_min(nlo, make_float4(other(nlo.x), other(nlo.y), other(nlo.z), 0.f));
            nhi = box_max(nhi, make_float4(other(nhi.x), other(nhi.y), other(nhi.z), 0.f));
        }
        const float ctr[3] = {0.5f * (nlo.x + nhi.x), 0.5f * (nlo.y + nhi.y), 0.5f * (nlo.z + nhi.z)};
        const double dc[3] = {0.5 * (double(lo.x) + hi.x) - ctr[0], 0.5 * (double(lo.y) + hi.y) - ctr[1],
                              0.5 * (double(lo.z) + hi.z) - ctr[2]};
        // as integers of the same order: the assignment compares them some 70 times (+ 0.0: -0 is 0)
        unsigned long long cost[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            double c = (t & 1) ? -dc[0] : dc[0];
            c += (t & 2) ? -dc[1] : dc[1];
            c += (t & 4) ? -dc[2] : dc[2];
            const long long bits = __double_as_longlong(c + 0.0);
            cost[t] = static_cast<unsigned long long>(bits) ^ (bits < 0 ? ~0ull : 1ull << 63);
        }
        uint32_t taken = 0u;         // slots given out
        unsigned long long map = 0;  // slot -> child, a byte each
        bool placed = ch < 0;
        for (int k = 0; k < nch; k++) {
            // the smallest cost over unplaced children and free slots, ties to the smaller child, then slot
            unsigned long long bc = ~0ull;
            int bi = s, bs = 8;
#pragma unroll
            for (int t = 0; t < 8; t++)
                if (!placed && !((taken >> t) & 1u) && cost[t] < bc) {
                    bc = cost[t];
                    bs = t;
                }
            if (bs == 8) bi = 8;  // nothing to offer
            for (int o = 1; o < 8; o <<= 1) {
                const unsigned long long oc = __shfl_xor_sync(gm, bc, o);
                const int oi = __shfl_xor_sync(gm, bi, o), os = __shfl_xor_sync(gm, bs, o);
                if (oc < bc || (oc == bc && oi < bi)) {
                    bc = oc;
                    bi = oi;
                    bs = os;
                }
            }
            if (bi > 7) { bad = true; break; }  // no finite cost is left (the same in all lanes)
            taken |= 1u << bs;
            map |= static_cast<unsigned long long>(bi) << (8 * bs);
            if (s == bi) placed = true;
        }
        if (bad) {
            atomicOr(&E.st->now.err, kErrLayout);
            continue;
        }
        // lane s takes over the child of slot s
        const bool valid = (taken >> s) & 1u;
        const int src = valid ? int((map >> (8 * s)) & 0xffu) : s;
        lo = make_float4(from(lo.x, src), from(lo.y, src), from(lo.z, src), 0.f);
        hi = make_float4(from(hi.x, src), from(hi.y, src), from(hi.z, src), 0.f);
        ch = from(ch, src);
        cnt = from(cnt, src);
        leaf = from(int(leaf), src) != 0;
        const bool is_leaf = valid && leaf;
        const uint32_t imask = (__ballot_sync(gm, valid && !leaf) >> (lane & 24)) & 0xffu;
        // slots for internal children (contiguous wide nodes) and leaf triangles (contiguous records)
        const int mine = is_leaf ? cnt : 0;
        int off = mine;
        for (int o = 1; o < 8; o <<= 1) {
            const int v = __shfl_up_sync(gm, off, o, 8);
            if (s >= o) off += v;
        }
        const int nint = __popc(imask), ntri = from(off, 7);
        off -= mine;
        int32_t child_base = 0, tri_base = 0;
        if (s == 0) {
            child_base = nint ? atomicAdd(&E.st->now.wide_count, nint) : 0;
            tri_base = ntri ? atomicAdd(&E.st->tri_count, ntri) : 0;
        }
        child_base = from(child_base, 0);
        tri_base = from(tri_base, 0);
        if (__any_sync(gm, child_base + nint > E.wide_cap || (is_leaf && (cnt < 1 || cnt > kMaxLeaf || off > 31)))) {
            atomicOr(&E.st->now.err, kErrLayout);
            continue;
        }
        uint32_t meta = 0u;
        if (valid && !leaf) {
            meta = 0x80u;
            E.q_bin[child_base + __popc(imask & ((1u << s) - 1u))] = ch;
        } else if (is_leaf) {
            meta = uint32_t((cnt << 5) | off);
            // the leaf's triangles, left to right
            int32_t st[8];
            int sp = 0;
            st[sp++] = ch;
            int32_t rec = tri_base + off;
            while (sp > 0) {
                const int32_t m = st[--sp];
                if (N.left[m] < 0) {
                    const int32_t t = N.right[m];
                    const float* p = E.P + 9 * int64_t(t);
                    const float p1x = p[0], p1y = p[1], p1z = p[2];
                    E.tris[size_t(rec) * 3] = make_float4(p1x, p1y, p1z, __fsub_rn(p[3], p1x));
                    E.tris[size_t(rec) * 3 + 1] = make_float4(__fsub_rn(p[4], p1y), __fsub_rn(p[5], p1z), __fsub_rn(p[6], p1x),
                                                              __fsub_rn(p[7], p1y));
                    E.tris[size_t(rec) * 3 + 2] = make_float4(__fsub_rn(p[8], p1z), __uint_as_float(uint32_t(t)), 0.f, 0.f);
                    E.tri_slot[t] = rec;
                    rec++;
                    continue;
                }
                if (sp + 2 > 8) { bad = true; break; }
                st[sp++] = N.right[m];
                st[sp++] = N.left[m];
            }
        }
        __syncwarp(gm);
        // Quantization (bvh_build.cpp quantize), with the margin check in double: lo, hi and p are
        // floats and q * 2^(eb-127) a multiple of the quantum, which the exponent choice keeps within
        // 2^-45 of |p|, so p + q * quantum is exact in double.
        uint32_t eb[3];
        float origin[3];
        uint32_t ql[3], qh[3];
        const float nl[3] = {nlo.x, nlo.y, nlo.z}, nh[3] = {nhi.x, nhi.y, nhi.z};
        const float bl[3] = {lo.x, lo.y, lo.z}, bh[3] = {hi.x, hi.y, hi.z};
        bool quantized = true;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double ext = double(nh[a]) - double(nl[a]);
            const double mag = fmax(fabs(double(nl[a])), fabs(double(nh[a])));
            bool ok = false;
            for (int e = max(exponent_for(ext / 251.0), exponent_for(mag * 1.2e-7)); e <= 254 && !ok; e++) {
                // the quantum and its inverse, both powers of two (the product is the quotient)
                const double q = __hiloint2double((e - 127 + 1023) << 20, 0), iq = __hiloint2double((127 - e + 1023) << 20, 0);
                const double pd = double(nl[a]) - 2.0 * q;
                float p = __double2float_rn(pd);
                if (double(p) > pd) p = nextafterf(p, -INFINITY);
                bool fits = double(p) < double(nl[a]) - q;
                uint32_t l8 = 255u, h8 = 0u;  // an empty slot's inverted box
                if (fits && valid) {
                    const double l = floor((double(bl[a]) - double(p)) * iq) - 1.0, h = ceil((double(bh[a]) - double(p)) * iq) + 1.0;
                    fits = !(l < 0.0 || h > 255.0) && !(double(p) + l * q + q > double(bl[a]) || double(p) + h * q - q < double(bh[a]));
                    if (fits) {
                        l8 = uint32_t(l);
                        h8 = uint32_t(h);
                    }
                }
                ok = __all_sync(gm, fits);
                if (ok) {
                    eb[a] = uint32_t(e);
                    origin[a] = p;
                    ql[a] = l8;
                    qh[a] = h8;
                }
            }
            quantized = quantized && ok;
        }
        if (__any_sync(gm, bad)) {
            atomicOr(&E.st->now.err, kErrLayout);
            continue;
        }
        if (!quantized) {  // the same in all lanes of the group
            atomicOr(&E.st->now.err, kErrQuantize);
            continue;
        }
        // four slots' bytes per word: lanes 0-3 the first, 4-7 the second
        auto word = [&](uint32_t v) {
            v <<= 8 * (s & 3);
            v |= __shfl_xor_sync(gm, v, 1);
            return v | __shfl_xor_sync(gm, v, 2);
        };
        uint32_t* o = E.nodes + size_t(w) * 20;
        const uint32_t mw = word(meta);
        uint32_t lw[3], hw[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            lw[a] = word(ql[a]);
            hw[a] = word(qh[a]);
        }
        if (s == 0) {
            o[0] = fbits(origin[0]); o[1] = fbits(origin[1]); o[2] = fbits(origin[2]);
            o[3] = eb[0] | (eb[1] << 8) | (eb[2] << 16) | (imask << 24);
            o[4] = uint32_t(child_base);
            o[5] = uint32_t(tri_base);
        }
        if ((s & 3) == 0) {
            const int half = s >> 2;
            o[6 + half] = mw;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                o[8 + 2 * a + half] = lw[a];
                o[14 + 2 * a + half] = hw[a];
            }
        }
    }
}

// Level 0: the root's wide node.
__global__ void k_emit_start(Emit E) {
    E.q_bin[0] = E.root->root;
    E.st->now.wide_count = 1;
    E.st->tri_count = 0;
    E.st->level[0] = LevelEnd{0, 0};
    E.st->level[1] = LevelEnd{1, 0};
}

int grid_of(int64_t n) { return int(std::min<int64_t>((n + kBlock - 1) / kBlock, int64_t(1) << 20)); }

}  // namespace gpubuild

// Builds into device buffers: `nodes` (20 words per wide node), `tris` (12 floats per record),
// `tri_slot` (flattened index -> record). Synchronous on `st`.
void build_bvh8_gpu(const float* tri_p, int64_t n, DevBuf& nodes, DevBuf& tris, DevBuf& tri_slot, int64_t& num_nodes,
                    int32_t& depth, double& sah_cost, cudaStream_t st) {
    using namespace gpubuild;
    if (n <= 0) throw Error(LMGPU_ERR_INVALID_ARGUMENT, "accel build: no triangles");
    if (n > (int64_t(1) << 30)) throw Error(LMGPU_ERR_UNSUPPORTED, "accel build: more than 2^30 triangles on the GPU builder");
    const size_t nn = size_t(2) * size_t(n);
    const int width = std::min(8, std::max(2, tuning().node_width));
    // One allocation holds every temporary (26 of them, with their releases, took most of a small
    // build's time).
    size_t sort_bytes = 0;
    {
        cub::DoubleBuffer<uint32_t> dk(nullptr, nullptr);
        cub::DoubleBuffer<int32_t> dv(nullptr, nullptr);
        LMGPU_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, dk, dv, int(n), 0, 30, st));
    }
    struct Part {
        void** p;
        size_t bytes;
    };
    float *P, *cost;
    float4 *tlo, *thi, *cen, *blo, *bhi;
    uint32_t *cb, *keys[2];
    int32_t *vals[2], *bl, *br, *bc, *cl[2], *nnb, *q;
    int8_t *dec, *dnode;
    unsigned long long* sums;
    void* tmp;
    PlocState* state;
    RootInfo* root;
    EmitState* es;
    auto at = [](auto*& p) { return reinterpret_cast<void**>(&p); };
    const Part parts[] = {
        {at(P), size_t(n) * 36}, {at(tlo), size_t(n) * 16}, {at(thi), size_t(n) * 16}, {at(cen), size_t(n) * 16},
        {at(cb), 24}, {at(keys[0]), size_t(n) * 4}, {at(keys[1]), size_t(n) * 4}, {at(vals[0]), size_t(n) * 4},
        {at(vals[1]), size_t(n) * 4}, {at(blo), nn * 16}, {at(bhi), nn * 16}, {at(bl), nn * 4}, {at(br), nn * 4},
        {at(bc), nn * 4}, {at(cost), nn * 32}, {at(dec), nn * 8}, {at(dnode), nn}, {at(cl[0]), size_t(n) * 4},
        {at(cl[1]), size_t(n) * 4}, {at(nnb), size_t(n) * 4}, {at(sums), (size_t(n) / kBlock + 1) * 8},
        {at(q), size_t(n) * 4}, {&tmp, sort_bytes}, {at(state), 2 * sizeof(PlocState)},
        {at(root), sizeof(RootInfo)}, {at(es), sizeof(EmitState)}};
    size_t total = 0;
    for (const Part& x : parts) total += (x.bytes + 255) & ~size_t(255);
    DevBuf arena;
    arena.alloc(total);
    {
        char* p = arena.as<char>();
        for (const Part& x : parts) {
            *x.p = p;
            p += (x.bytes + 255) & ~size_t(255);
        }
    }
    LMGPU_CUDA(cudaMemcpyAsync(P, tri_p, size_t(n) * 36, cudaMemcpyHostToDevice, st));
    LMGPU_CUDA(cudaMemsetAsync(cb, 0xff, 12, st));  // ordered minima, then maxima
    LMGPU_CUDA(cudaMemsetAsync(cb + 3, 0, 12, st));
    LMGPU_CUDA(cudaMemsetAsync(es, 0, sizeof(EmitState), st));
    const int g = grid_of(n);
    k_prep<<<g, kBlock, 0, st>>>(P, n, tlo, thi, cen, cb, &es->now.err);
    k_morton<<<g, kBlock, 0, st>>>(cen, n, cb, keys[0], vals[0]);
    LMGPU_CUDA(cudaGetLastError());
    cub::DoubleBuffer<uint32_t> dk(keys[0], keys[1]);
    cub::DoubleBuffer<int32_t> dv(vals[0], vals[1]);
    LMGPU_CUDA(cub::DeviceRadixSort::SortPairs(tmp, sort_bytes, dk, dv, int(n), 0, 30, st));
    const Nodes N{blo, bhi, bl, br, bc, cost, dec, dnode};
    k_leaves<<<g, kBlock, 0, st>>>(dv.Current(), n, tlo, thi, N, cl[0], state);
    LMGPU_CUDA(cudaGetLastError());

    int herr = 0;
    auto check = [&] {
        if (herr & kErrNonFinite) throw Error(LMGPU_ERR_INVALID_ARGUMENT, "accel build: non-finite vertex coordinate");
        if (herr & kErrQuantize) throw Error(LMGPU_ERR_INVALID_ARGUMENT, "accel build: box quantization failed");
        if (herr) throw Error(LMGPU_ERR_INTERNAL, "accel build: internal error (wide node layout)");
    };

    // PLOC: passes over all clusters, four between two reads of what is left (a pass leaves about three
    // quarters; blocks past the end leave at once), then the last ones in one block
    int cur = 0, iters = 0;
    for (int32_t m = int32_t(n); m > kLast;) {
        const int gm = int((m + kBlock - 1) / kBlock);
        for (int k = 0; k < 4; k++, cur = 1 - cur) {
            k_nearest<<<gm, kBlock, 0, st>>>(cl[cur], state + cur, N.lo, N.hi, nnb, sums);
            k_scan_blocks<<<1, 1024, 0, st>>>(sums, gm, state + cur, state + 1 - cur);
            k_merge<<<gm, kBlock, 0, st>>>(cl[cur], state + cur, nnb, sums, N, cl[1 - cur], width);
            LMGPU_CUDA(cudaGetLastError());
        }
        PlocState h{};
        LMGPU_CUDA(cudaMemcpyAsync(&h, state + cur, sizeof(h), cudaMemcpyDeviceToHost, st));
        LMGPU_CUDA(cudaMemcpyAsync(&herr, &es->now.err, 4, cudaMemcpyDeviceToHost, st));
        LMGPU_CUDA(cudaStreamSynchronize(st));
        check();
        if (h.m < 1 || h.m >= m || h.next_id - int32_t(n) != int32_t(n) - h.m)
            throw Error(LMGPU_ERR_INTERNAL, "accel build: clustering made no progress");
        m = h.m;
        if (++iters > 100000) throw Error(LMGPU_ERR_INTERNAL, "accel build: clustering did not converge");
    }
    k_last_passes<<<1, kLast, 0, st>>>(cl[cur], state + cur, N, width, root, &es->now.err);
    LMGPU_CUDA(cudaGetLastError());
    // Non-finite input is refused here at the latest: from the allocations below on, the tree that the
    // outputs may still hold is overwritten. The wait replaces the one for the root at the end.
    RootInfo hr{};
    LMGPU_CUDA(cudaMemcpyAsync(&hr, root, sizeof(hr), cudaMemcpyDeviceToHost, st));
    LMGPU_CUDA(cudaMemcpyAsync(&herr, &es->now.err, 4, cudaMemcpyDeviceToHost, st));
    LMGPU_CUDA(cudaStreamSynchronize(st));
    check();

    // emission, four levels between two reads of how many nodes there are
    num_nodes = 0;  // until it is done the outputs hold no tree
    const int32_t cap = int32_t(std::max<int64_t>(n, 1));  // wide nodes never exceed the triangles
    nodes.alloc(size_t(cap) * 80);
    tris.alloc(size_t(n) * 48);
    tri_slot.alloc(size_t(n) * 4);
    const Emit E{N, P, nodes.as<uint32_t>(), tris.as<float4>(), tri_slot.as<int32_t>(), q, es, root, cap, width};
    k_emit_start<<<1, 1, 0, st>>>(E);
    LMGPU_CUDA(cudaGetLastError());
    EmitState h{};
    int32_t levels = 0;
    const int emit_grid = int(std::min<int64_t>((n + kEmitBlock / 8 - 1) / (kEmitBlock / 8), int64_t(current_device().num_sms) * 16));
    auto empty = [&](int32_t l) { return h.level[l & 7].wide_count == h.level[(l + 1) & 7].wide_count; };
    do {
        for (int k = 0; k < 4; k++, levels++) {
            k_emit<<<emit_grid, kEmitBlock, 0, st>>>(E, levels);
            LMGPU_CUDA(cudaGetLastError());
            LMGPU_CUDA(cudaMemcpyAsync(&es->level[(levels + 2) & 7], &es->now, sizeof(LevelEnd), cudaMemcpyDeviceToDevice, st));
        }
        LMGPU_CUDA(cudaMemcpyAsync(&h, es, sizeof(h), cudaMemcpyDeviceToHost, st));
        LMGPU_CUDA(cudaStreamSynchronize(st));
        herr = h.now.err;
        check();
    } while (!empty(levels));
    while (levels > 0 && empty(levels - 1)) levels--;
    if (int64_t(h.tri_count) != n) throw Error(LMGPU_ERR_INTERNAL, "accel build: internal error (triangle count)");
    const double dx = double(hr.hi[0]) - hr.lo[0], dy = double(hr.hi[1]) - hr.lo[1], dz = double(hr.hi[2]) - hr.lo[2];
    const double ra = 2.0 * (dx * dy + dy * dz + dz * dx);
    sah_cost = ra > 0 ? double(hr.cost) / ra : 0.0;
    num_nodes = h.now.wide_count;
    depth = levels;
}

}  // namespace lmgpu
