// The warp's work loop with a pool of leaves (trace_batch_pool): what a node step finds is tested by any lane.
#pragma once

#include "traverse.cuh"

namespace dipl {

// A lane's ray for the node steps.
struct NodeRay {
    float3 o, inv;
    float tmin;
};

constexpr int kStepLeaves = 4;   // leaf references a lane's node step yields at most
constexpr int kLeafPool = 31 + 32 * kStepLeaves;  // at most 31 leaves stay, and a step adds the rest

// The rays a block works on, one column per ray (the thread it started on), and per warp the leaves to be tested.
template <int LEAF, bool ANY>
struct PoolRays {
    // origin, tmin, direction (watertight: the shear, and its axes as bits); one word per column, so that lanes which read
    // any columns of their warp meet no bank twice
    float state[LEAF == DIPL_LEAF_WATERTIGHT ? 8 : 7][kTraceThreads];
    float4 hit[ANY ? 1 : kTraceThreads];              // closest hit: t, u, v, primitive
    unsigned long long best[ANY ? 1 : kTraceThreads];  // its order: ordered bits of t above the primitive
    float tmax[ANY ? kTraceThreads : 1];
    unsigned open[ANY ? kTraceThreads : 1];            // any hit: 0 once hit
    int lanes[kTraceThreads];    // lanes at work on the ray
    long long ray[kTraceThreads];
    uint32_t leaves[kTraceThreads / 32];       // in the warp's pool
    int2 leaf[kTraceThreads / 32][kLeafPool];  // leaf reference, column of its ray
};

// The work of a warp on a batch, laid over rays as in trace_batch. There a lane holds the leaves it meets and 10 of 32
// lanes test a triangle at a time, while the others wait with theirs or for a node. Here a node step puts its leaves into
// a pool of the warp, and lanes test any of them, 32 at a time or as many as there are lanes with a node left: 31 lanes
// work in a node step and 30 in a test (4M-triangle soup, 2M rays: 206 + 110 steps of a warp, before about 350 + 340),
// and the node step keeps no leaf test's state. A ray's column in shared memory has what a test needs and its closest
// hit, which the least (t, primitive) wins; a lane is done with a ray once its last leaf has been tested.
// Was against lanes that hold their leaves: 8-wide 2M-triangle soup, 2M sorted rays 10.1 -> 8.6 ms, 1M sphere, 4M rays 384
// -> 356 us; 4-wide occlusion of a soup, 1M rays 1018 -> 926 us, 512 x 512 frame with shadows 602 -> 511 us. Bound by issue
// slots (75%, about 290 instructions a step). Leaves by ballots instead of the pool's atomic count: 8-wide soup -3%,
// frame +3%, occlusion +3%. A lane waiting once it has one or two leaves in the pool: +4 to +10%; tests at half as many
// leaves: +5%. The layout's steps `v` (one object per lane):
//   clear(), begin(ray)   no work; the root as the lane's work
//   has_node()            a node to visit next, or leaves of one that are not in the pool yet
//   node(ray, lim, bot, lf)  one step; up to kStepLeaves leaf references come back in lf (0: none); the stack is used down
//                         to `bot`
//   sp, kShort, steps, bad, take(ray, thread, entry, column)  as in trace_batch
//   kRoundedInverse       load_ray's ROUNDED
template <int LEAF, bool ANY, bool PERSIST, class V>
__device__ __forceinline__ void trace_batch_pool(V& v, PoolRays<LEAF, ANY>& S, const float4* __restrict__ tris, bool backface,
                                            const Batch& B) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
    const uint32_t lt_mask = lanemask_lt();
    const int64_t warp_id = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int2* const pool = S.leaf[threadIdx.x >> 5];
    NodeRay r{};
    int col = threadIdx.x;   // the column of this lane's ray
    int count = 0;           // leaves in the pool (warp-uniform)
    uint32_t tested = 0;     // leaves tested so far (warp-uniform): the pool holds the leaves from there on
    uint32_t last = 0;       // one past this lane's last leaf
    auto position = [&](int64_t k) -> int64_t { return (((k >> 5) * warps + warp_id) << 5) + (k & 31); };
    int64_t next = 0;   // rays this warp has taken (warp-uniform)
    bool working = false;  // this lane has a ray
    auto start_ray = [&](int64_t cand) {
        const int64_t my = B.order ? (int64_t)__ldg(B.order + cand) : cand;  // the ray's own index (hits go there)
        const RayState q = load_ray<V::kRoundedInverse>(B.rays, my);
        working = true;
        S.ray[threadIdx.x] = my;
        r.o = q.o, r.inv = q.inv, r.tmin = q.tmin;
        float3 e = q.d;
        if (LEAF == DIPL_LEAF_WATERTIGHT) {
            const WtRay w = wt_setup(q.d);
            e = make_float3(w.sx, w.sy, w.sz);
            S.state[7 % (sizeof(S.state) / sizeof(S.state[0]))][threadIdx.x] = __int_as_float(w.kx | (w.ky << 2) | (w.kz << 4));
        }
        const float state[7] = {q.o.x, q.o.y, q.o.z, q.tmin, e.x, e.y, e.z};
#pragma unroll
        for (int k = 0; k < 7; ++k) S.state[k][threadIdx.x] = state[k];
        if (ANY) {
            S.open[threadIdx.x] = 1u;
            S.tmax[threadIdx.x] = q.tmax;
        } else {
            S.hit[threadIdx.x] = make_float4(__int_as_float(0x7F800000), 0.0f, 0.0f, __int_as_float(-1));
            S.best[threadIdx.x] = (unsigned long long)ordered_bits(q.tmax + 0.0f) << 32;
        }
        last = tested;
        v.steps = 0;
        v.clear();
        // A ray that cannot hit anything under either leaf test (an empty interval, an origin that is not finite or a
        // NaN direction: t then comes out NaN or beyond kInfinity) does no work.
        const bool live = q.tmax > q.tmin && isfinite(q.o.x) && isfinite(q.o.y) && isfinite(q.o.z) && !isnan(q.d.x) &&
                          !isnan(q.d.y) && !isnan(q.d.z);
        if (live && !B.empty) v.begin(r);
    };
    auto limit = [&]() {
        return ANY ? prune_limit(S.tmax[col])
                   : prune_limit(from_ordered_bits((unsigned)(S.best[col] >> 32)));
    };
    // Tests the pool's leaves while there are `least` of them, 32 at a time.
    auto test_leaves = [&](int least) {
        int head = 0;
        while (count - head >= least && head < count) {
            __syncwarp();
            int c = 0, i = 0, n = 0;
            if (head + lane < count) {
                const int2 e = pool[head + lane];
                c = e.y;
                i = leaf_first(e.x), n = leaf_count(e.x);  // an unused child slot has no triangles
            }
            for (;;) {
                unsigned long long key = ~0ull;
                float t = 0.0f, b1 = 0.0f, b2 = 0.0f;
                int prim = -1;
                if (n > 0) {
                    float4 p0, p1, p2;
                    load_leaf_triangle(tris, i, p0, p1, p2);
                    const float3 o = make_float3(S.state[0][c], S.state[1][c], S.state[2][c]);
                    const float3 d = make_float3(S.state[4][c], S.state[5][c], S.state[6][c]);
                    const float3 pa = make_float3(p0.x, p0.y, p0.z), pb = make_float3(p1.x, p1.y, p1.z),
                                 pc = make_float3(p2.x, p2.y, p2.z);
                    if (LEAF == DIPL_LEAF_WATERTIGHT) {
                        const int axes = __float_as_int(S.state[7 % (sizeof(S.state) / sizeof(S.state[0]))][c]);
                        const WtRay w{axes & 3, (axes >> 2) & 3, axes >> 4, d.x, d.y, d.z};
                        t = wt_test(pa, pb, pc, o, w, backface, b1, b2);
                    } else {
                        t = mt_ref(pa, pb, pc, o, d, backface, b1, b2);
                    }
                    // t == kInfinity is the tests' miss value (also when tmax is +inf)
                    if (t > S.state[3][c] && t < kInfinity) {
                        if (ANY) {
                            if (t < S.tmax[c]) S.open[c] = 0u;
                        } else {
                            const int id = __float_as_int(p0.w);
                            key = ((unsigned long long)ordered_bits(t + 0.0f) << 32) | (unsigned)id;
                            // Only what is below the word may win it: as it starts, it equals the key of primitive 0 at
                            // t == tmax, which is no hit.
                            if (key < S.best[c]) {
                                prim = id;
                                atomicMin(&S.best[c], key);
                            }
                        }
                    }
                    --n, ++i;
                }
                if (!ANY) {
                    __syncwarp();
                    if (prim >= 0 && S.best[c] == key) S.hit[c] = make_float4(t, b1, b2, __int_as_float(prim));
                }
                if (!__any_sync(full, n > 0)) break;
                __syncwarp();  // this round's reads and records before the next round's minima
            }
            head += 32;
        }
        if (head) {
            head = min(head, count);
            tested += head;
            count -= head;
            __syncwarp();
            int2 e;
            if (lane < count) e = pool[head + lane];
            __syncwarp();
            if (lane < count) pool[lane] = e;
            if (lane == 0) S.leaves[threadIdx.x >> 5] = count;
            __syncwarp();
        }
    };
    // One step of the warp (called by all lanes; `on`: this lane has work): a node for every lane that has one, whose
    // leaves go to the pool.
    auto warp_step = [&](bool on, int bot) {
        int lf[kStepLeaves] = {};
        if (on && v.has_node()) {
            if (++v.steps > B.step_limit) v.bad = true, v.clear();
            else v.node(r, limit(), bot, lf);
        }
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < kStepLeaves; ++k) c += lf[k] != 0 ? 1u : 0u;
        v.steps += c;
        if (c) {
            int at = (int)atomicAdd(&S.leaves[threadIdx.x >> 5], c);
            last = tested + at + c;
#pragma unroll
            for (int k = 0; k < kStepLeaves; ++k)
                if (lf[k]) pool[at++] = make_int2(lf[k], col);
        }
        __syncwarp();
        count = (int)S.leaves[threadIdx.x >> 5];
        __syncwarp();  // read by every lane, before the next step counts on
        const uint32_t nodes = __ballot_sync(full, on && v.has_node());
        const int least = max(1, __popc(nodes));
        if (count >= least) test_leaves(least);
        if (ANY && on && S.open[col] == 0u) v.clear();
    };
    auto busy = [&]() { return v.has_node() || (int32_t)(last - tested) > 0; };
    auto write_hit = [&](int column) {
        const int64_t i = S.ray[column];
        if (ANY) {
            B.occluded[i] = S.open[column] == 0u ? 1 : 0;
        } else {
            const float4 h = S.hit[column];
            reinterpret_cast<int4*>(B.hits)[i] = make_int4(__float_as_int(h.w), __float_as_int(h.x), __float_as_int(h.y),
                                                           __float_as_int(h.z));
        }
    };

    if (lane == 0) S.leaves[threadIdx.x >> 5] = 0;
    __syncwarp();
    // ---- every lane its own ray --------------------------------------------------------------------------------
    v.clear();
    if (!PERSIST) {
        const int64_t cand = warp_id * B.group + lane;
        if (lane < B.group && cand < B.n) start_ray(cand);
    }
    for (;;) {
        bool more = false;
        if (PERSIST) {
            const uint32_t idle = __ballot_sync(full, !working);
            more = position(next) < B.n;
            if (more && __popc(idle) >= kRefillLanes) {
                if (!working) {
                    const int64_t cand = position(next + __popc(idle & lt_mask));
                    if (cand < B.n) start_ray(cand);
                }
                next += __popc(idle);
                more = position(next) < B.n;
            }
        }
        const uint32_t active = __ballot_sync(full, working);
        if (!more && __popc(active) <= kShareLanes) break;
        warp_step(working, 0);
        if (working && !busy()) {
            write_hit(threadIdx.x);
            working = false;
        }
    }

    // ---- the warp's last rays, shared by its lanes -----------------------------------------------------------------
    // A lane without work takes the bottom stack entry (the largest pending subtree) of a lane that has one, with that
    // lane's ray; the last lane on a ray writes its record. Entries leave a stack at the bottom (bot) only while they
    // are in shared memory.
    int bot = 0;
    if (working) S.lanes[threadIdx.x] = 1;
    for (;;) {
        __syncwarp();  // the last step's shared-memory writes, before other lanes read them
        const uint32_t idle = __ballot_sync(full, !working);
        if (idle == full) break;
        const bool can_give = working && v.sp > bot && bot < V::kShort;
        const uint32_t givers = __ballot_sync(full, can_give);
        if (idle && givers) {
            const int rank = __popc(idle & lt_mask);
            const bool take = !working && rank < __popc(givers);
            const int src = take ? nth_set_bit(givers, rank) : lane;
            const int sbot = __shfl_sync(full, bot, src), scol = __shfl_sync(full, col, src);
            NodeRay q;
            q.inv.x = __shfl_sync(full, r.inv.x, src), q.inv.y = __shfl_sync(full, r.inv.y, src);
            q.inv.z = __shfl_sync(full, r.inv.z, src);
            const uint32_t ssteps = __shfl_sync(full, v.steps, src);
            if (take) {
                col = scol;
                q.o = make_float3(S.state[0][col], S.state[1][col], S.state[2][col]);
                q.tmin = S.state[3][col];
                r = q;
                v.steps = ssteps;
                v.clear();
                bot = 0;
                last = tested;
                v.take(r, wbase + src, sbot, col);
                working = true;
                atomicAdd(&S.lanes[col], 1);
            }
            __syncwarp();  // entries read, before their lanes overwrite them
            if (can_give && __popc(givers & lt_mask) < __popc(idle)) {
                ++bot;
                if (bot == v.sp) bot = v.sp = 0;
            }
        }
        warp_step(working, bot);
        __syncwarp();
        if (working && !busy()) {
            if (atomicSub(&S.lanes[col], 1) == 1) write_hit(col);
            working = false;
        }
    }
    if (v.bad) atomicOr(B.err, kErrStack);
}

// The lane's work for layouts whose children are references to nodes (>= 0) and leaves (< 0): a node `cur` (kRefIdle:
// none) and a stack of nodes, whose first kShort entries live in shared memory, one column per thread, the rest in local
// memory. The layout adds begin, take and node.
template <int STACK, int SHORT>
struct RefStack {
    static constexpr int kShort = SHORT;
    static constexpr bool kRoundedInverse = false;
    int* column;  // this thread's stack column
    int* rest;    // entries from SHORT on: an array of the kernel's (inside this object it would keep the rest in memory)
    int root, num_nodes;
    bool bad = false;
    int cur = kRefIdle;
    uint32_t steps = 0;
    int sp = 0;

    __device__ __forceinline__ bool has_node() const { return cur != kRefIdle; }
    __device__ __forceinline__ void clear() { cur = kRefIdle, sp = 0; }
    __device__ __forceinline__ void put(int at, int ref) {
        if (at < SHORT) column[at * kTraceThreads] = ref;
        else rest[at - SHORT] = ref;
    }
    __device__ __forceinline__ void pop(int bot) {
        cur = kRefIdle;
        if (sp > bot) {
            --sp;
            cur = column[min(sp, SHORT - 1) * kTraceThreads];
            if (sp >= SHORT) cur = rest[sp - SHORT];
        }
    }
    // An entry of another lane's stack.
    __device__ __forceinline__ int entry_of(int thread, int entry) const {
        return column[entry * kTraceThreads + thread - (int)threadIdx.x];
    }
    // False, with the step done, when cur is no node: a root that is a leaf, or a corrupted tree.
    __device__ __forceinline__ bool check(int pushes, int (&lf)[kStepLeaves]) {
        if ((unsigned)cur < (unsigned)num_nodes && sp + pushes <= STACK) return true;
        if (cur < 0) lf[0] = cur;
        else bad = true;
        cur = kRefIdle;
        return false;
    }
};

}  // namespace dipl
