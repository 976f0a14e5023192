// What the trace kernels share: rays, leaf tests, and the warp's work loop (trace_batch) over a layout's own steps.
#pragma once

#include <algorithm>

#include "internal.h"
#include "intersect.cuh"

namespace dipl {

constexpr int kTraceThreads = 128;
constexpr float kPruneSlack = 1e-5f;

struct RayState {
    float3 o, d, inv;
    float tmin, tmax;
};

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One 32-byte read-only load (p must be 32-byte aligned): a 64-byte node in two loads instead of four.
__device__ __forceinline__ void ldg_v8(const void* p, float4& x, float4& y) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w)
        : "l"(p));
}

// ROUNDED: reciprocals rounded to nearest, those of directions above 8.5e37 subnormal (0 otherwise).
template <bool ROUNDED = false>
__device__ __forceinline__ RayState load_ray(const dipl_ray* rays, int64_t i) {
    const float4* r4 = reinterpret_cast<const float4*>(rays) + 2 * i;
    const float4 a = __ldg(r4), b = __ldg(r4 + 1);
    RayState r;
    r.o = make_float3(a.x, a.y, a.z);
    r.d = make_float3(b.x, b.y, b.z);
    r.tmin = a.w;
    r.tmax = b.w;
    // Directions below 1e-20 in magnitude are treated as +-1e-20 so that 1/d stays finite and a ray lying
    // on a slab plane is still inside it (0 * inf would be NaN). 1/d only feeds the slab tests, which widen
    // their interval by 1e-6 relative: the hardware reciprocal (relative error below 2^-22) is well inside
    // that margin.
    auto safe = [](float x) { return fabsf(x) < 1e-20f ? copysignf(1e-20f, x) : x; };
    auto rcp = [](float x) { return ROUNDED ? __frcp_rn(x) : rcp_approx(x); };
    r.inv = make_float3(rcp(safe(r.d.x)), rcp(safe(r.d.y)), rcp(safe(r.d.z)));
    return r;
}

__device__ __forceinline__ float prune_limit(float best_t) { return best_t + fabsf(best_t) * kPruneSlack; }

// Float bits in an order that compares like the floats (for warp minima).
__device__ __forceinline__ unsigned ordered_bits(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Triangle i's three float4 in two loads: records are 48 bytes, so either the first or the last 32 bytes of a record
// are aligned for a 32-byte load.
__device__ __forceinline__ void load_leaf_triangle(const float4* __restrict__ tris, int i, float4& p0, float4& p1,
                                                   float4& p2) {
    const float4* tp = tris + 3 * (int64_t)i;
    const bool odd = i & 1;
    float4 a, b;
    ldg_v8(tp + (odd ? 1 : 0), a, b);
    const float4 c = __ldg(tp + (odd ? 0 : 2));
    p0 = odd ? c : a;
    p1 = odd ? a : b;
    p2 = odd ? b : c;
}

// A lane's ray and the best hit it has found. best_t starts at tmax (an any-hit ray keeps it).
template <int LEAF, bool ANY>
struct LaneRay {
    float3 o, d, inv;
    float tmin;
    WtRay w;
    float best_t, best_u, best_v;
    int best_prim;
    bool found;

    // False when the ray cannot hit anything under either leaf test: an empty interval, an origin that is not finite
    // or a NaN direction (t then comes out NaN or beyond kInfinity).
    __device__ __forceinline__ bool start(const dipl_ray* rays, int64_t i) {
        const RayState r = load_ray(rays, i);
        o = r.o, d = r.d, inv = r.inv, tmin = r.tmin;
        reset(r.tmax);
        return r.tmax > r.tmin && isfinite(r.o.x) && isfinite(r.o.y) && isfinite(r.o.z) && !isnan(r.d.x) &&
               !isnan(r.d.y) && !isnan(r.d.z);
    }
    __device__ __forceinline__ void reset(float tmax) {
        if (LEAF == DIPL_LEAF_WATERTIGHT) w = wt_setup(d);
        best_t = tmax, best_u = 0.0f, best_v = 0.0f, best_prim = -1, found = false;
    }
    __device__ __forceinline__ void test(const float4* __restrict__ tris, int i, bool backface) {
        float4 p0, p1, p2;
        load_leaf_triangle(tris, i, p0, p1, p2);
        const int prim = __float_as_int(p0.w);
        const float3 a = make_float3(p0.x, p0.y, p0.z), b = make_float3(p1.x, p1.y, p1.z),
                     c = make_float3(p2.x, p2.y, p2.z);
        float b1 = 0.0f, b2 = 0.0f;
        const float t = LEAF == DIPL_LEAF_REF_MT ? mt_ref(a, b, c, o, d, backface, b1, b2)
                                                 : wt_test(a, b, c, o, w, backface, b1, b2);
        // t == kInfinity is the tests' miss value (also when tmax is +inf)
        if (ANY) {
            if (t > tmin && t < best_t && t < kInfinity) found = true;
        } else if (t > tmin && t < kInfinity && (t < best_t || (t == best_t && found && prim < best_prim))) {
            best_t = t, best_u = b1, best_v = b2, best_prim = prim, found = true;
        }
    }
};

// A warp whose rays have all started shares the last of them among its lanes once at most this many lanes have one
// (24: 512x512 frame +2%, 8: 8-wide soup +3%, 0: 1M sphere 0.63 against 0.37 ms, 64k rays there 152 against 62 us).
constexpr int kShareLanes = 16;
constexpr int kLeafTurn = 8;     // lanes that hold a leaf before triangles are tested (1 to 16: within 1%, 24: -5%)
constexpr int kRefillLanes = 4;  // idle lanes before a persistent warp takes new rays (1: +3%, 16: +10%)

// Rays shared by a warp, one column per ray (the lane it started on).
template <bool ANY>
struct SharedRays {
    float4 best[ANY ? 1 : kTraceThreads];  // closest hit of the lanes that are done: t, u, v, primitive
    float tmax[ANY ? 1 : kTraceThreads];
    unsigned lim[kTraceThreads];           // ordered bits of the least t of all lanes; any hit: 0 once hit
    int lanes[kTraceThreads];              // lanes at work on the ray
    long long ray[kTraceThreads];          // the ray's index
};

struct Batch {
    const dipl_ray* rays;
    int64_t n;
    dipl_hit* hits;
    uint8_t* occluded;
    const uint32_t* order;  // the ray at each position of the work order (nullptr: as given)
    uint32_t* err;
    uint32_t step_limit;
    int group;              // one-shot: rays per warp
    bool empty;             // no nodes and no triangles
};

// The work of a warp on a batch. PERSIST: a grid of resident warps that walk the batch together, a warp's k-th ray at
// position ((k / 32) * warps + warp) * 32 + k % 32; idle lanes take new rays. Otherwise warp w has the `group` rays from
// w * group on. The layout's steps `v` (one object per lane):
//   begin(ray)            the root as the lane's work
//   has_node(), has_leaf()  a node to visit next; triangles to test
//   node(ray, lim, bot), leaf(ray, bot)  one step: a node or a triangle; the stack is used down to `bot`
//   drop()                no more work; bad: a step found the tree corrupt or a limit passed
//   sp, kShort            stack entries; those below kShort are in shared memory
//   take(ray, thread, entry, owner)  entry of the stack of the block's thread `thread` as the lane's work; `owner`: the
//                         thread on which the ray started
template <int LEAF, bool ANY, bool PERSIST, class V>
__device__ __forceinline__ void trace_batch(V& v, LaneRay<LEAF, ANY>& r, SharedRays<ANY>& S, const Batch& B) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
    const uint32_t lt_mask = lanemask_lt();
    const int64_t warp_id = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    auto position = [&](int64_t k) -> int64_t { return (((k >> 5) * warps + warp_id) << 5) + (k & 31); };
    int64_t next = 0;   // rays this warp has taken (warp-uniform)
    int64_t my = -1;    // this lane's ray, -1 when idle
    float tmax = 0.0f;
    auto start_ray = [&](int64_t cand) {
        my = B.order ? (int64_t)__ldg(B.order + cand) : cand;  // the ray's own index (hits go there)
        const bool live = r.start(B.rays, my);
        tmax = r.best_t;
        v.steps = 0;
        v.sp = 0;
        v.drop();
        if (live && !B.empty) v.begin(r);
    };
    auto busy = [&]() { return v.has_node() || v.has_leaf(); };
    // One step of the warp (called by all lanes; `on`: this lane has work): a node for every lane that has one, then,
    // once kLeafTurn lanes hold a leaf or no lane has a node left, a triangle for every lane that holds a leaf. True
    // when triangles were tested.
    auto warp_step = [&](bool on, float lim, int bot) {
        if (on && v.has_node()) {
            if (++v.steps > B.step_limit) v.bad = true, v.drop();
            else v.node(r, lim, bot);
        }
        const uint32_t holds = __ballot_sync(full, on && v.has_leaf());
        const uint32_t nodes = __ballot_sync(full, on && v.has_node());
        if (holds == 0u || (nodes != 0u && __popc(holds) < kLeafTurn)) return false;
        if (on && v.has_leaf()) {
            if (++v.steps > B.step_limit) v.bad = true, v.drop();
            else v.leaf(r, bot);
            if (ANY && r.found) v.drop();
        }
        return true;
    };
    auto write_hit = [&](int64_t i, float t, float u, float vv, int prim) {
        reinterpret_cast<int4*>(B.hits)[i] =
            prim >= 0 ? make_int4(prim, __float_as_int(t), __float_as_int(u), __float_as_int(vv))
                      : make_int4(-1, 0x7F800000, 0, 0);
    };

    // ---- every lane its own ray --------------------------------------------------------------------------------
    v.drop();
    if (!PERSIST) {
        const int64_t cand = warp_id * B.group + lane;
        if (lane < B.group && cand < B.n) start_ray(cand);
    }
    for (;;) {
        bool more = false;
        if (PERSIST) {
            const uint32_t idle = __ballot_sync(full, my < 0);
            more = position(next) < B.n;
            if (more && __popc(idle) >= kRefillLanes) {
                if (my < 0) {
                    const int64_t cand = position(next + __popc(idle & lt_mask));
                    if (cand < B.n) start_ray(cand);
                }
                next += __popc(idle);
                more = position(next) < B.n;
            }
        }
        const uint32_t active = __ballot_sync(full, my >= 0);
        if (!more && __popc(active) <= kShareLanes) break;
        warp_step(my >= 0, prune_limit(r.best_t), 0);
        if (my >= 0 && !busy()) {
            if (ANY) B.occluded[my] = r.found ? 1 : 0;
            else write_hit(my, r.best_t, r.best_u, r.best_v, r.found ? r.best_prim : -1);
            my = -1;
        }
    }

    // ---- the warp's last rays, shared by its lanes -----------------------------------------------------------------
    // A lane without work takes the bottom stack entry (the largest pending subtree) of a lane that has one, with that
    // lane's ray. Lanes prune by the least t any lane has found for the ray (lim) but accept hits against their own,
    // so that the smallest (t, primitive id) of all lanes is the record a single lane would produce; each lane that
    // runs out of work merges its best, and the last one writes the record. Entries leave a stack at the bottom (bot)
    // only while they are in shared memory.
    int owner = lane, bot = 0;
    bool working = my >= 0;
    if (working) {
        S.ray[threadIdx.x] = my;
        S.lanes[threadIdx.x] = 1;
        S.lim[threadIdx.x] = ANY ? 1u : ordered_bits(r.best_t);
        if (!ANY) {
            S.tmax[threadIdx.x] = tmax;
            S.best[threadIdx.x] = r.found ? make_float4(r.best_t, r.best_u, r.best_v, __int_as_float(r.best_prim))
                                          : make_float4(__int_as_float(0x7F800000), 0.0f, 0.0f, __int_as_float(-1));
        }
    }
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
            const int sbot = __shfl_sync(full, bot, src), sowner = __shfl_sync(full, owner, src);
            float3 qo, qd, qi;
            qo.x = __shfl_sync(full, r.o.x, src), qo.y = __shfl_sync(full, r.o.y, src);
            qo.z = __shfl_sync(full, r.o.z, src), qd.x = __shfl_sync(full, r.d.x, src);
            qd.y = __shfl_sync(full, r.d.y, src), qd.z = __shfl_sync(full, r.d.z, src);
            qi.x = __shfl_sync(full, r.inv.x, src), qi.y = __shfl_sync(full, r.inv.y, src);
            qi.z = __shfl_sync(full, r.inv.z, src);
            const float qmin = __shfl_sync(full, r.tmin, src);
            const uint32_t ssteps = __shfl_sync(full, v.steps, src);
            const float qmax = ANY ? __shfl_sync(full, r.best_t, src) : 0.0f;
            if (take) {
                owner = sowner;
                r.o = qo, r.d = qd, r.inv = qi, r.tmin = qmin;
                r.reset(ANY ? qmax : S.tmax[wbase + owner]);
                v.steps = ssteps;
                v.sp = bot = 0;
                v.take(r, wbase + src, sbot, wbase + owner);
                working = true;
                atomicAdd(&S.lanes[wbase + owner], 1);
            }
            __syncwarp();  // entries read, before their lanes overwrite them
            if (can_give && __popc(givers & lt_mask) < __popc(idle)) {
                ++bot;
                if (bot == v.sp) bot = v.sp = 0;
            }
        }
        const unsigned lb = working ? S.lim[wbase + owner] : 0u;
        if (ANY && working && lb == 0u) v.drop();
        const float before = r.best_t;
        if (warp_step(working, prune_limit(ANY ? r.best_t : from_ordered_bits(lb)), bot) && working) {
            if (ANY) {
                if (r.found) S.lim[wbase + owner] = 0u;
            } else if (r.best_t < before) {
                atomicMin(&S.lim[wbase + owner], ordered_bits(r.best_t));
            }
        }
        uint32_t done = __ballot_sync(full, working && !busy());
        while (done) {  // one lane at a time: several may have worked on one ray
            if (lane == __ffs(done) - 1) {
                const int o = wbase + owner;
                if (!ANY && r.found) {
                    const float4 b = S.best[o];
                    if (r.best_t < b.x || (r.best_t == b.x && (unsigned)r.best_prim < (unsigned)__float_as_int(b.w)))
                        S.best[o] = make_float4(r.best_t, r.best_u, r.best_v, __int_as_float(r.best_prim));
                }
                const int left = S.lanes[o] - 1;
                S.lanes[o] = left;
                if (left == 0) {
                    if (ANY) {
                        B.occluded[S.ray[o]] = S.lim[o] == 0u ? 1 : 0;
                    } else {
                        const float4 b = S.best[o];
                        write_hit(S.ray[o], b.x, b.y, b.z, __float_as_int(b.w));
                    }
                }
                working = false;
            }
            done &= done - 1u;
            __syncwarp();
        }
    }
    if (v.bad) atomicOr(B.err, kErrStack);
}

// The lane's work as references to nodes and leaf ranges, for layouts whose children are such references: a node
// (cur >= 0), kRefIdle, or a leaf (cur < 0) that waits for `held` to be taken; `held`: the leaf range whose triangles
// are tested next, 0 for none; a stack of references whose first kShort entries live in shared memory, one column per
// thread, the rest in local memory. The layout adds begin, take and node.
constexpr int kRefPop = -0x7FFFFFFF - 1;  // next: pop the stack
constexpr int kRefIdle = 0x7FFFFFFF;      // no node

template <int STACK, int SHORT>
struct RefWork {
    static constexpr int kShort = SHORT;
    const float4* tris;
    int* column;  // this thread's stack column
    int root;
    bool backface;
    bool bad = false;
    int cur = kRefIdle, held = 0;
    uint32_t steps = 0;
    int sp = 0;
    int* rest;  // entries from SHORT on: an array of the kernel's (inside this object it would keep the rest in memory)

    __device__ __forceinline__ bool has_node() const { return cur >= 0 && cur != kRefIdle; }
    __device__ __forceinline__ bool has_leaf() const { return held != 0; }
    __device__ __forceinline__ void drop() { cur = kRefIdle, held = 0; }
    __device__ __forceinline__ void enter(int ref) {
        cur = ref, held = 0;
        if (ref < 0) held = ref, cur = kRefIdle;
    }
    __device__ __forceinline__ void put(int at, int ref) {
        if (at < SHORT) column[at * kTraceThreads] = ref;
        else rest[at - SHORT] = ref;
    }
    __device__ __forceinline__ void push(int ref) { put(sp++, ref); }
    __device__ __forceinline__ int pop(int bot) {
        int ref = kRefIdle;
        if (sp > bot) {
            --sp;
            ref = column[min(sp, SHORT - 1) * kTraceThreads];
            if (sp >= SHORT) ref = rest[sp - SHORT];
        }
        return ref;
    }
    // After cur was entered (or set to kRefPop): a leaf moves to a free `held`, and cur is popped where it is empty. Two
    // pops at most: the second leaf waits in cur.
    __device__ __forceinline__ void advance(int bot) {
        if (cur == kRefPop) cur = pop(bot);
        if (cur < 0 && held == 0) {
            held = cur;
            cur = pop(bot);
        }
    }
    template <class R>
    __device__ __forceinline__ void leaf(R& r, int bot) {
        const int first = leaf_first(held), cnt = leaf_count(held);
        if (cnt > 0) r.test(tris, first, backface);  // an unused child slot has no triangles
        held = cnt > 1 ? make_leaf_ref(first + 1, cnt - 1) : 0;
        advance(bot);
    }
};

// Blocks of a persistent trace launch: every resident block on every SM (per kernel instantiation and device).
template <auto Kernel>
int persistent_grid() {
    static DeviceProbe probe;  // per instantiation
    return probe_per_device(probe, [] {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Kernel, kTraceThreads, 0);
        (void)cudaGetLastError();
        return std::max(1, sms * std::max(1, per_sm));
    });
}

// Steps one ray may take: at most one per node and one per leaf triangle.
inline uint32_t steps_bound(int64_t nodes, int64_t triangles) {
    return trace_step_limit() ? trace_step_limit()
                              : (uint32_t)std::min<int64_t>(0xFFFFFFFFll, 2 * std::max<int64_t>(nodes, 0) + triangles + 64);
}

// How a batch is laid over the kernels ONE (one-shot) and MANY (persistent) of one layout; launch(kernel, grid, group).
// Batches that the resident lanes hold at once are spread over all warps, down to one ray per warp, whose other
// lanes then share it (4096 rays of a small frame: 28 us, 60 with 32 rays per warp). Larger ones in the given order
// run on resident warps that refill idle lanes, since their rays may differ most in length (1M sphere, 4M rays
// 0.38 ms against 1.11 with one ray per lane; 1M occlusion rays 1.17 against 1.69; where all rays are alike one
// ray per lane is a little faster: 1M primary rays 0.41 against 0.36). Sorted rays get one lane each: a warp's
// rays are then of similar length and start together (4M-triangle soup 11.2 against 13.8 ms). Both sides of each pair
// with the 4-wide nodes and held leaves.
template <auto ONE, auto MANY, class L>
void launch_batch(int64_t n, bool sorted, L&& launch) {
    const int64_t warps = (int64_t)persistent_grid<ONE>() * (kTraceThreads / 32);
    if (!sorted && n > warps * 32) {
        launch(MANY, (unsigned)persistent_grid<MANY>(), 32);
    } else {
        const int group = (int)std::min<int64_t>(32, std::max<int64_t>(1, (n + warps - 1) / warps));
        const int64_t per_block = (int64_t)group * (kTraceThreads / 32);
        launch(ONE, (unsigned)((n + per_block - 1) / per_block), group);
    }
}

}  // namespace dipl
