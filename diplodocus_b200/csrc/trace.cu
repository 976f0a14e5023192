// Closest-hit and any-hit traversal of the binary layout. Traces walk its 4-wide nodes (quad_trace_kernel); counted
// traces walk the binary FP32 nodes themselves, whose visits the counters report (trace_kernel, tail_kernel).
//
// Replaces SBvh::Intersect / IntersectAny (src/acceleration/sbvh.cc:60-191) and the device brute force
// DummyIntersect / DummyIntersectAny (src/gpu/renderer/gpu_renderer_util.h:29-94).
//
// Closest-hit rule: among triangles with tmin < t < tmax, the smallest t, ties to the lowest primitive id.
// That is exactly what the reference brute force returns (ascending ids, strict <,
// dummy_acceleration_structure.cc:21-64). To keep it under any traversal order the box tests are
// conservative: slab distances widen by 1e-6 relative (their own rounding, with the approximate reciprocal
// of the direction, stays below 5e-7), boxes are padded
// by 2^-20 of their coordinate magnitude at build time, and a node is pruned only when it starts beyond
// the best t by more than 1e-5 relative, so a node can never be skipped for rounding of its own box.
#include <limits>

#include "internal.h"
#include "intersect.cuh"

namespace dipl {
namespace {

constexpr int kTraceThreads = 128;
// Resident blocks per SM the kernel is compiled for: 9 x 128 threads at <= 56 registers. Builds with more
// registers and 8 blocks per SM measured up to 1.5x slower on the 16M-triangle soup.
constexpr int kTraceMinBlocks = 9;
constexpr float kSlabWiden = 1e-6f;
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
    r.inv = make_float3(rcp_approx(safe(r.d.x)), rcp_approx(safe(r.d.y)), rcp_approx(safe(r.d.z)));
    return r;
}

// Conservative ray/box interval; returns entry t (or +inf when the box is missed or out of range).
__device__ __forceinline__ float box_entry(const RayState& r, float lx, float hx, float ly, float hy, float lz, float hz,
                                           float t_limit) {
    const float tx0 = __fmul_rn(__fsub_rn(lx, r.o.x), r.inv.x), tx1 = __fmul_rn(__fsub_rn(hx, r.o.x), r.inv.x);
    const float ty0 = __fmul_rn(__fsub_rn(ly, r.o.y), r.inv.y), ty1 = __fmul_rn(__fsub_rn(hy, r.o.y), r.inv.y);
    const float tz0 = __fmul_rn(__fsub_rn(lz, r.o.z), r.inv.z), tz1 = __fmul_rn(__fsub_rn(hz, r.o.z), r.inv.z);
    float tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
    float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
    tn = tn - fabsf(tn) * kSlabWiden;
    tf = tf + fabsf(tf) * kSlabWiden;
    const bool hit = tn <= tf && tf >= r.tmin && tn <= t_limit;
    return hit ? tn : __int_as_float(0x7F800000);
}

__device__ __forceinline__ float prune_limit(float best_t) { return best_t + fabsf(best_t) * kPruneSlack; }

// Traversal stack of (node reference, entry t). Entries [0, SHORT) live in shared memory, one column per
// thread (entry k of thread j at sh[k * kTraceThreads + j], so a warp's accesses never share a bank), the rest
// in local memory.
template <int STACK, int SHORT>
struct Stack {
    int2* sh;
    int ref[STACK - SHORT];
    float t[STACK - SHORT];
    int sp = 0;
    __device__ __forceinline__ void push(int r, float tt) {
        if (sp < SHORT) {
            sh[sp * kTraceThreads] = make_int2(r, __float_as_int(tt));
        } else {
            ref[sp - SHORT] = r;
            t[sp - SHORT] = tt;
        }
        ++sp;
    }
    __device__ __forceinline__ int2 get(int k) const {
        return k < SHORT ? sh[k * kTraceThreads] : make_int2(ref[k - SHORT], __float_as_int(t[k - SHORT]));
    }
};

// Long rays of a warp that has no rays left to take move to tail_kernel: once at most kTailLanes lanes of the warp
// are still tracing, a lane whose ray has taken kTailSteps steps or more writes the ray's state (ray index, next
// node, best hit so far, stack) to a slot and takes no more work; tail_kernel then traverses each such ray with a
// whole warp. Without it the warp keeps issuing one-lane steps until its longest ray ends (the 1M sphere's
// grazing rays take up to ~430 steps). With all 32 lanes busy (the soup) nothing is offloaded: the warp is
// already fully used. Measured (4M rays on the 1M sphere / 1M rays on the 16M soup, identical hits): 0.633 ->
// 0.497 ms / 52.97 -> 51.85 ms; offloading at 8-32 steps sends rays whose remaining work is too short for a
// warp (sphere 0.73-0.84 ms), and offloading from full warps slows the soup (55.2 ms).
constexpr int kTailSteps = 64;
constexpr int kTailLanes = 8;  // ... and only when at most this many lanes of the warp are still tracing
constexpr int kTailHeaderInts = 12;  // ray (2), cur, sp, best t/u/v, prim, found, pad
constexpr size_t kTailBytes = 64u << 20;  // slot storage per trace call, at most
// Batches smaller than this trace without the offload: their warps run out of rays early, the rays of
// such batches are mostly short (a 512x512 frame of the small scene), and the offload's allocation, clearing
// and extra launch cost more there (0.243 against 0.279-0.289 ms per frame of two traces).
constexpr int64_t kTailMinRays = 1 << 19;

struct TailQueue {
    int* slots;          // slot_ints ints each: header, then sp (ref, t) pairs
    unsigned* count;     // [0]: slots written (may exceed cap), [1]: slots taken by tail_kernel
    int cap;             // slots available
    int slot_ints;
    int min_steps;       // 0: no offload
    int max_lanes;
    uint32_t step_limit; // steps one ray may take (both kernels), beyond which it is given up and flagged
};

// Float bits in an order that compares like the floats (for warp minima).
__device__ __forceinline__ unsigned ordered_bits(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Leaf test dispatch: ref_mt or watertight.
template <int LEAF>
__device__ __forceinline__ float leaf_test(float3 a, float3 b, float3 c, const RayState& r, const WtRay& w,
                                           bool backface, float& b1, float& b2) {
    if (LEAF == DIPL_LEAF_REF_MT) return mt_ref(a, b, c, r.o, r.d, backface, b1, b2);
    return wt_test(a, b, c, r.o, w, backface, b1, b2);
}

// Counted traversal: every lane advances its ray by one inner node or one leaf triangle per step. With a persistent grid
// (rays in the given order) a lane whose ray finished takes its warp's next ray at the following step, so lanes do
// not idle behind the warp's longest ray (most rays of a batch may finish at the root while a few descend to the
// leaves); with one lane per ray (the coherent order) each warp traces its 32 rays and hands long ones on.
template <int LEAF, int STACK, int SHORT>
__global__ void __launch_bounds__(kTraceThreads, kTraceMinBlocks) trace_kernel(const BNode* __restrict__ nodes,
                                                              const float4* __restrict__ tris, int root,
                                                              int num_nodes, const dipl_ray* __restrict__ rays,
                                                              int64_t n, dipl_hit* __restrict__ hits, uint32_t flags,
                                                              unsigned long long* __restrict__ counters,
                                                              uint32_t* __restrict__ err, TailQueue tq,
                                                              const uint32_t* __restrict__ order) {
    __shared__ int2 sh_stack[SHORT > 0 ? SHORT * kTraceThreads : 1];
    const int lane = threadIdx.x & 31;
    const int64_t warp_id = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    // The k-th ray a warp takes is at position ((k / 32) * warps + warp) * 32 + k % 32 of the work order, so all
    // warps walk the order together and the rays in flight are one window of it (a coherent order then keeps the
    // whole GPU in one region of the tree; one chunk per warp measured 181 against 163 ms on the pre-split soup).
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t end = n;
    auto position = [&](int64_t k) -> int64_t { return (((k >> 5) * warps + warp_id) << 5) + (k & 31); };
    const bool backface = (flags & DIPL_TRACE_BACKFACE_CULLING) != 0u;
    const uint32_t lt_mask = lanemask_lt();
    const uint32_t step_limit = tq.step_limit;
    int64_t next = 0;    // rays this warp has taken (warp-uniform)
    int64_t my = -1;     // this lane's ray, -1 when idle
    RayState r{};
    WtRay w{};
    float best_t = 0.0f, best_u = 0.0f, best_v = 0.0f;
    int best_prim = -1;
    bool found = false;
    int cur = 0;
    uint32_t steps = 0;
    Stack<STACK, SHORT> st;
    st.sh = sh_stack + threadIdx.x;
    unsigned visits = 0, tests = 0;
    bool bad = false;
    bool may_offload = tq.min_steps > 0;
    for (;;) {
        // ---- refill idle lanes ---------------------------------------------------------------------
        const bool idle = my < 0;
        const uint32_t idle_mask = __ballot_sync(0xffffffffu, idle);
        if (idle_mask) {
            if (idle) {
                const int64_t cand = position(next + __popc(idle_mask & lt_mask));
                if (cand < end) {
                    my = order ? (int64_t)__ldg(order + cand) : cand;  // the ray's own index (hits go there)
                    r = load_ray(rays, my);
                    if (LEAF == DIPL_LEAF_WATERTIGHT) w = wt_setup(r.d);
                    best_t = r.tmax, best_u = 0.0f, best_v = 0.0f, best_prim = -1, found = false;
                    cur = num_nodes >= 0 ? root : 0x7FFFFFFF;
                    st.sp = 0;
                    steps = 0;
                }
            }
            if (position(next) < end) next += __popc(idle_mask);
        }
        const uint32_t active_mask = __ballot_sync(0xffffffffu, my >= 0);
        if (!active_mask) break;
        if (my < 0) continue;

        // ---- one step: an inner node or a leaf --------------------------------------------------------
        bool finished = false;
        if (cur == 0x7FFFFFFF) {
            finished = true;  // empty BVH
        } else if (++steps > step_limit || (cur >= 0 && cur >= num_nodes)) {
            bad = true;       // only a corrupted tree gets here
            finished = true;
        } else if (cur >= 0) {
            const float4* np = reinterpret_cast<const float4*>(nodes + cur);
            float4 a, b, c, df;
            ldg_v8(np, a, b);
            ldg_v8(np + 2, c, df);
            const int2 d = make_int2(__float_as_int(df.x), __float_as_int(df.y));
            ++visits;
            const float lim = prune_limit(best_t);
            const float t0 = box_entry(r, a.x, a.y, a.z, a.w, c.x, c.y, lim);
            const float t1 = box_entry(r, b.x, b.y, b.z, b.w, c.z, c.w, lim);
            const bool h0 = t0 != __int_as_float(0x7F800000), h1 = t1 != __int_as_float(0x7F800000);
            if (h0 && h1) {
                const bool first0 = t0 <= t1;
                if (st.sp >= STACK) {
                    bad = true;
                    finished = true;
                } else {
                    st.push(first0 ? d.y : d.x, first0 ? t1 : t0);
                    cur = first0 ? d.x : d.y;
                }
            } else if (h0) {
                cur = d.x;
            } else if (h1) {
                cur = d.y;
            } else {
                cur = -0x7FFFFFFF - 1;  // pop below
            }
        } else if (cur != -0x7FFFFFFF - 1) {
            // one triangle per step: a lane at a leaf never holds the warp for the leaf's other triangles (the
            // rest of the leaf stays in cur as the reference of its remaining triangles)
            const int first = leaf_first(cur), cnt = leaf_count(cur);
            const float4* tp = tris + 3 * (int64_t)first;
            const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
            const int prim = __float_as_int(p0.w);
            float b1 = 0.0f, b2 = 0.0f;
            const float t = leaf_test<LEAF>(make_float3(p0.x, p0.y, p0.z), make_float3(p1.x, p1.y, p1.z),
                                            make_float3(p2.x, p2.y, p2.z), r, w, backface, b1, b2);
            ++tests;
            // t == kInfinity is the tests' miss value (also when tmax is +inf)
            if (t > r.tmin && t < kInfinity && (t < best_t || (t == best_t && found && prim < best_prim))) {
                best_t = t;
                best_prim = prim;
                best_u = b1;
                best_v = b2;
                found = true;
            }
            if (cnt > 1) cur = make_leaf_ref(first + 1, cnt - 1);
            else cur = -0x7FFFFFFF - 1;  // pop below
        }
        if (!finished && cur == -0x7FFFFFFF - 1) {
            // pop the next entry that can still hold a better hit
            const float lim = prune_limit(best_t);
            cur = 0x7FFFFFFF;
            while (st.sp > 0) {
                --st.sp;
                const int2 e = st.get(st.sp);
                if (__int_as_float(e.y) <= lim) {
                    cur = e.x;
                    break;
                }
            }
            if (cur == 0x7FFFFFFF) finished = true;
        }
        if (finished) {
            int4 out;
            out.x = found ? best_prim : -1;
            out.y = __float_as_int(found ? best_t : __int_as_float(0x7F800000));
            out.z = __float_as_int(found ? best_u : 0.0f);
            out.w = __float_as_int(found ? best_v : 0.0f);
            reinterpret_cast<int4*>(hits)[my] = out;
            my = -1;
        } else if (may_offload && position(next) >= end && steps >= (uint32_t)tq.min_steps &&
                   __popc(active_mask) <= tq.max_lanes) {
            // the warp has no rays left and this ray is still going: hand it to tail_kernel if a slot is free
            const unsigned slot = atomicAdd(&tq.count[0], 1u);
            if (slot < (unsigned)tq.cap) {
                int* w = tq.slots + (size_t)slot * tq.slot_ints;
                w[0] = (int)(uint32_t)(uint64_t)my;
                w[1] = (int)(uint32_t)((uint64_t)my >> 32);
                w[2] = cur;
                w[3] = st.sp;
                w[4] = __float_as_int(best_t);
                w[5] = __float_as_int(best_u);
                w[6] = __float_as_int(best_v);
                w[7] = best_prim;
                w[8] = found ? 1 : 0;
                for (int k = 0; k < st.sp; ++k) reinterpret_cast<int2*>(w + kTailHeaderInts)[k] = st.get(k);
                my = -1;
            }
            may_offload = false;  // one try per lane
        }
    }
    if (bad) atomicOr(err, kErrStack);
    const unsigned v = __reduce_add_sync(0xffffffffu, visits);
    const unsigned t = __reduce_add_sync(0xffffffffu, tests);
    if (lane == 0) {
        atomicAdd(&counters[0], (unsigned long long)v);
        atomicAdd(&counters[1], (unsigned long long)t);
    }
}

// One warp per offloaded ray. Its pending work (the node it was at and its stack entries) is dealt round-robin to
// the lanes; each lane traverses near-child first with its own stack, lanes without work take the bottom entry
// (the largest pending subtree) of a lane holding two or more, and every step prunes against the best t of the
// whole warp (warp minimum, the same conservative slack as the main kernel). Each lane accepts leaf hits by the
// closest-hit rule against its own best; the warp then keeps the smallest (t, primitive id) over its lanes and
// the hit carried over from the main kernel, so the record is the one a single thread would produce.
template <int LEAF, int STACK>
__global__ void __launch_bounds__(kTraceThreads) tail_kernel(const BNode* __restrict__ nodes,
                                                             const float4* __restrict__ tris, int num_nodes,
                                                             const dipl_ray* __restrict__ rays,
                                                             dipl_hit* __restrict__ hits, uint32_t flags,
                                                             unsigned long long* __restrict__ counters,
                                                             uint32_t* __restrict__ err, TailQueue tq) {
    constexpr int kNone = -0x7FFFFFFF - 1;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t lt_mask = lanemask_lt();
    const bool backface = (flags & DIPL_TRACE_BACKFACE_CULLING) != 0u;
    const uint32_t step_limit = tq.step_limit;
    const unsigned total = min(*reinterpret_cast<volatile unsigned*>(&tq.count[0]), (unsigned)tq.cap);
    if (total == 0) return;  // nothing was handed on: the whole grid leaves at once
    unsigned visits = 0, tests = 0;
    bool bad = false;
    int sref[STACK];
    float stt[STACK];
    for (;;) {
        // slots claimed one at a time: a warp that drew a short ray takes the next (a fixed warp stride
        // measured slower on the 1M sphere, 0.525 against 0.50 ms)
        unsigned slot = 0;
        if (lane == 0) slot = atomicAdd(&tq.count[1], 1u);
        slot = __shfl_sync(full, slot, 0);
        if (slot >= total) break;
        const int* w = tq.slots + (size_t)slot * tq.slot_ints;
        const int64_t my = (int64_t)(((uint64_t)(uint32_t)w[1] << 32) | (uint32_t)w[0]);
        const int sp0 = min(w[3], STACK);
        const RayState r = load_ray(rays, my);
        WtRay wt{};
        if (LEAF == DIPL_LEAF_WATERTIGHT) wt = wt_setup(r.d);
        float best_t = r.tmax, best_u = 0.0f, best_v = 0.0f;
        int best_prim = -1;
        bool found = false;
        if (lane == 0 && w[8]) {
            best_t = __int_as_float(w[4]), best_u = __int_as_float(w[5]), best_v = __int_as_float(w[6]);
            best_prim = w[7];
            found = true;
        }
        // deal the pending items: stack entries 0..sp0-1, then the node the ray was at (always visited)
        int bot = 0, sp = 0, cur = kNone;
        for (int k = lane; k <= sp0; k += 32) {
            int ref;
            float t;
            if (k < sp0) {
                const int2 e = reinterpret_cast<const int2*>(w + kTailHeaderInts)[k];
                ref = e.x, t = __int_as_float(e.y);
            } else {
                ref = w[2], t = -__int_as_float(0x7F800000);
            }
            sref[sp] = ref, stt[sp] = t, ++sp;
        }
        uint32_t steps = 0;
        for (;;) {
            const float gbest = from_ordered_bits(__reduce_min_sync(full, ordered_bits(best_t)));
            const float lim = prune_limit(gbest);
            while (cur == kNone && sp > bot) {
                --sp;
                if (stt[sp] <= lim) cur = sref[sp];
            }
            if (sp == bot) sp = bot = 0;
            const bool hungry = cur == kNone;
            const uint32_t hm = __ballot_sync(full, hungry);
            if (hm == full) break;
            if (hm) {
                const uint32_t dm = __ballot_sync(full, sp - bot >= 2);
                const int nh = __popc(hm), nd = __popc(dm);
                const bool donate = ((dm >> lane) & 1u) && __popc(dm & lt_mask) < nh;
                int gref = kNone;
                float gt = 0.0f;
                if (donate) {
                    gref = sref[bot], gt = stt[bot];
                    ++bot;
                }
                const int rank = __popc(hm & lt_mask);
                const bool receive = hungry && rank < nd;
                const int src = receive ? nth_set_bit(dm, rank) : lane;
                const int rref = __shfl_sync(full, gref, src);
                const float rt = __shfl_sync(full, gt, src);
                if (receive && rref != kNone && rt <= lim) cur = rref;
            }
            if (cur != kNone) {
                if (++steps > step_limit || (cur >= 0 && cur >= num_nodes)) {
                    bad = true;
                    cur = kNone;
                    sp = bot = 0;
                } else if (cur >= 0) {
                    const float4* np = reinterpret_cast<const float4*>(nodes + cur);
                    float4 a, b, c, df;
                    ldg_v8(np, a, b);
                    ldg_v8(np + 2, c, df);
                    ++visits;
                    const float t0 = box_entry(r, a.x, a.y, a.z, a.w, c.x, c.y, lim);
                    const float t1 = box_entry(r, b.x, b.y, b.z, b.w, c.z, c.w, lim);
                    const bool h0 = t0 != __int_as_float(0x7F800000), h1 = t1 != __int_as_float(0x7F800000);
                    const int c0 = __float_as_int(df.x), c1 = __float_as_int(df.y);
                    if (h0 && h1) {
                        const bool first0 = t0 <= t1;
                        if (sp >= STACK) {
                            bad = true;
                            cur = kNone;
                        } else {
                            sref[sp] = first0 ? c1 : c0, stt[sp] = first0 ? t1 : t0, ++sp;
                            cur = first0 ? c0 : c1;
                        }
                    } else {
                        cur = h0 ? c0 : (h1 ? c1 : kNone);
                    }
                } else {
                    const int first = leaf_first(cur), cnt = leaf_count(cur);
                    for (int k = 0; k < cnt; ++k) {
                        const float4* tp = tris + 3 * (int64_t)(first + k);
                        const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                        const int prim = __float_as_int(p0.w);
                        float b1 = 0.0f, b2 = 0.0f;
                        const float t = leaf_test<LEAF>(make_float3(p0.x, p0.y, p0.z), make_float3(p1.x, p1.y, p1.z),
                                                        make_float3(p2.x, p2.y, p2.z), r, wt, backface, b1, b2);
                        ++tests;
                        if (t > r.tmin && t < kInfinity &&
                                   (t < best_t || (t == best_t && found && prim < best_prim))) {
                            best_t = t, best_prim = prim, best_u = b1, best_v = b2, found = true;
                        }
                    }
                    cur = kNone;
                }
            }
        }
        // the smallest (t, primitive id) of the warp
        const unsigned tk = found ? ordered_bits(best_t) : 0xFFFFFFFFu;
        const unsigned tmin = __reduce_min_sync(full, tk);
        const bool cand = found && tk == tmin;
        const unsigned pmin = __reduce_min_sync(full, cand ? (unsigned)best_prim : 0xFFFFFFFFu);
        const uint32_t win = __ballot_sync(full, cand && (unsigned)best_prim == pmin);
        const int wl = win ? __ffs(win) - 1 : 0;
        const float ft = __shfl_sync(full, best_t, wl), fu = __shfl_sync(full, best_u, wl),
                    fv = __shfl_sync(full, best_v, wl);
        const int fp = __shfl_sync(full, best_prim, wl);
        if (lane == 0) {
            int4 out;
            out.x = win ? fp : -1;
            out.y = __float_as_int(win ? ft : __int_as_float(0x7F800000));
            out.z = __float_as_int(win ? fu : 0.0f);
            out.w = __float_as_int(win ? fv : 0.0f);
            reinterpret_cast<int4*>(hits)[my] = out;
        }
    }
    if (bad) atomicOr(err, kErrStack);
    const unsigned v = __reduce_add_sync(full, visits);
    const unsigned t = __reduce_add_sync(full, tests);
    if (lane == 0) {
        atomicAdd(&counters[0], (unsigned long long)v);
        atomicAdd(&counters[1], (unsigned long long)t);
    }
}

// ---- 4-wide traversal -------------------------------------------------------------------------------------------
// Closest and any hits over QNodes. What bounds it: instruction issue and the L1 data pipe (one cycle per lane and
// load instruction, whatever its width), with a third to a half of the lanes idle because the lanes of a warp are at
// different kinds of work. Hence: nodes of 64 bytes in two loads for four children, triangles in two loads, a stack
// entry of one word (no entry distance: on the soup 96% of the popped entries are visited anyway, and the distances
// cost a third of the stack's shared memory and 1.3x of the time), one node or one triangle per lane and step, one
// leaf held back per lane so that it goes on with nodes until enough lanes of the warp hold one, and rays shared by
// all lanes of the warp when few are left. Measured against the binary traversal it replaces (node visits of the
// pre-split soup 359 -> 192 a ray, L1 cycles 1474 -> 760): 4M-triangle soup, 2M rays in the coherent order 15.2 ->
// 11.2 ms; 16M soup, 16M rays 127 -> 90 ms; 1M sphere, 4M rays 0.52 -> 0.38 ms; 4096 rays of a small frame 60 -> 28 us.
constexpr int kQPop = -0x7FFFFFFF - 1;   // next: pop the stack
constexpr int kQIdle = 0x7FFFFFFF;       // no node
constexpr float kQMiss = 3.40282346638528859812e+38f;  // entry distance of a child that is not entered
constexpr int kQShort = 32;              // stack entries per thread in shared memory: 24 with more blocks per SM and
                                         // 16 were slower (soup 12.2 and 12.9 against 11.3 ms)
// A warp whose rays have all started shares the last of them among its lanes once at most this many lanes have one
// (16 and 8 within 1%, 0: 1M sphere 0.63 against 0.37 ms, 64k rays there 152 against 62 us).
constexpr int kShareLanes = 24;
constexpr int kLeafTurn = 8;             // lanes that hold a leaf before triangles are tested (1 to 16: within 1%, 24: -5%)
constexpr int kRefillLanes = 4;          // idle lanes before a persistent warp takes new rays (1: +3%, 16: +10%)

struct QRay {
    float3 o, d, inv;
    float tmin;
};

// False when the ray cannot hit anything under either leaf test: an empty interval, an origin that is not finite or
// a NaN direction (t then comes out NaN or beyond kInfinity).
__device__ __forceinline__ bool quad_load_ray(const dipl_ray* rays, int64_t i, QRay& q, float& tmax) {
    const RayState r = load_ray(rays, i);
    q.o = r.o, q.d = r.d, q.inv = r.inv, q.tmin = r.tmin;
    tmax = r.tmax;
    return r.tmax > r.tmin && isfinite(r.o.x) && isfinite(r.o.y) && isfinite(r.o.z) && !isnan(r.d.x) &&
           !isnan(r.d.y) && !isnan(r.d.z);
}

// Traversal stack of references. The first kQShort entries live in shared memory, one column per thread (where the
// warp's other lanes can read them), the rest in local memory.
template <int STACK>
struct QStack {
    int* column;
    int rest[STACK - kQShort];
    int sp = 0;
    __device__ __forceinline__ void push_short(int ref) { column[sp++ * kTraceThreads] = ref; }
    __device__ __forceinline__ void push(int ref) {
        if (sp < kQShort) column[sp * kTraceThreads] = ref;
        else rest[sp - kQShort] = ref;
        ++sp;
    }
    __device__ __forceinline__ int pop() {
        --sp;
        return sp < kQShort ? column[sp * kTraceThreads] : rest[sp - kQShort];
    }
};

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

// Byte k of a plane word as the float 32768 + byte.
__device__ __forceinline__ float quad_plane(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7504u | (uint32_t)(k << 4)));
}

// The children of a node by entry distance (kQMiss when not entered), nearest first, and their references.
//
// A plane at p + Q s (Q = 32768 + byte) is met at t = (p - o) / d + Q (s / d). With a = p - o in FP32 and C = a / d
// the rounding of a and C is at most 2^-23 |C|; near planes move back and far planes on by 2^-22 |C|. What is
// relative to t (the reciprocal of d, the last FMA) stays below 2e-7 on either side and the final comparison allows
// 2e-6. A NaN plane (an overflowing product) does not constrain the interval.
__device__ __forceinline__ void quad_children(const QNode* __restrict__ quads, int node, const QRay& r, float lim,
                                              float (&key)[4], int (&ref)[4]) {
    float4 f0, f1, f2, f3;
    const float4* np = reinterpret_cast<const float4*>(quads + node);
    ldg_v8(np, f0, f1);
    ldg_v8(np + 2, f2, f3);
    ref[0] = __float_as_int(f1.x), ref[1] = __float_as_int(f1.y);
    ref[2] = __float_as_int(f1.z), ref[3] = __float_as_int(f1.w);
    const uint32_t eb = __float_as_uint(f0.w);  // the neighbouring exponent's low bit lands in the sign
    const float Sx = __fmul_rn(fabsf(__uint_as_float(eb << 23)), r.inv.x);
    const float Sy = __fmul_rn(fabsf(__uint_as_float((eb >> 8) << 23)), r.inv.y);
    const float Sz = __fmul_rn(fabsf(__uint_as_float((eb >> 16) << 23)), r.inv.z);
    const float Cx = __fmul_rn(__fsub_rn(f0.x, r.o.x), r.inv.x), Cy = __fmul_rn(__fsub_rn(f0.y, r.o.y), r.inv.y),
                Cz = __fmul_rn(__fsub_rn(f0.z, r.o.z), r.inv.z);
    constexpr float kE = 2.384185791015625e-07f;  // 2^-22
    const float nCx = __fmaf_rn(fabsf(Cx), -kE, Cx), fCx = __fmaf_rn(fabsf(Cx), kE, Cx);
    const float nCy = __fmaf_rn(fabsf(Cy), -kE, Cy), fCy = __fmaf_rn(fabsf(Cy), kE, Cy);
    const float nCz = __fmaf_rn(fabsf(Cz), -kE, Cz), fCz = __fmaf_rn(fabsf(Cz), kE, Cz);
    const uint32_t lx = __float_as_uint(f2.x), hx = __float_as_uint(f2.y), ly = __float_as_uint(f2.z),
                   hy = __float_as_uint(f2.w), lz = __float_as_uint(f3.x), hz = __float_as_uint(f3.y);
    const uint32_t nx = r.inv.x < 0.0f ? hx : lx, fx = r.inv.x < 0.0f ? lx : hx;
    const uint32_t ny = r.inv.y < 0.0f ? hy : ly, fy = r.inv.y < 0.0f ? ly : hy;
    const uint32_t nz = r.inv.z < 0.0f ? hz : lz, fz = r.inv.z < 0.0f ? lz : hz;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float tnx = __fmaf_rn(quad_plane(nx, k), Sx, nCx), tfx = __fmaf_rn(quad_plane(fx, k), Sx, fCx);
        const float tny = __fmaf_rn(quad_plane(ny, k), Sy, nCy), tfy = __fmaf_rn(quad_plane(fy, k), Sy, fCy);
        const float tnz = __fmaf_rn(quad_plane(nz, k), Sz, nCz), tfz = __fmaf_rn(quad_plane(fz, k), Sz, fCz);
        const float tn = fmaxf(max3(tnx, tny, tnz), r.tmin);
        const float tf = fminf(min3(tfx, tfy, tfz), lim);
        key[k] = tn <= __fmaf_rn(fabsf(tf), 2e-6f, tf) ? tn : kQMiss;
    }
    auto order = [&](int i, int j) {
        const bool swap = key[j] < key[i];
        const float a = swap ? key[j] : key[i], b = swap ? key[i] : key[j];
        const int c = swap ? ref[j] : ref[i], d = swap ? ref[i] : ref[j];
        key[i] = a, key[j] = b, ref[i] = c, ref[j] = d;
    };
    order(0, 1);
    order(2, 3);
    order(0, 2);
    order(1, 3);
    order(1, 2);
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

// PERSIST: a grid of resident warps that walk the batch together, a warp's k-th ray at position ((k / 32) * warps +
// warp) * 32 + k % 32; idle lanes take new rays. Otherwise warp w has the `group` rays from w * group on.
template <int LEAF, bool ANY, bool PERSIST, int STACK>
__global__ void __launch_bounds__(kTraceThreads, PERSIST ? 8 : 9) quad_trace_kernel(
    const QNode* __restrict__ quads, const float4* __restrict__ tris, int root, int num_nodes,
    const dipl_ray* __restrict__ rays, int64_t n, dipl_hit* __restrict__ hits, uint8_t* __restrict__ occluded,
    uint32_t flags, uint32_t* __restrict__ err, uint32_t step_limit, int group, const uint32_t* __restrict__ order) {
    const unsigned full = 0xffffffffu;
    __shared__ int sh_stack[kQShort * kTraceThreads];
    // rays shared by a warp, one column per ray (the lane it started on)
    __shared__ float4 s_best[ANY ? 1 : kTraceThreads];  // closest hit of the lanes that are done: t, u, v, primitive
    __shared__ float s_tmax[ANY ? 1 : kTraceThreads];
    __shared__ unsigned s_lim[kTraceThreads];           // ordered bits of the least t of all lanes; any hit: 0 once hit
    __shared__ int s_lanes[kTraceThreads];              // lanes at work on the ray
    __shared__ long long s_ray[kTraceThreads];          // the ray's index
    const int lane = threadIdx.x & 31, wbase = threadIdx.x & ~31;
    const uint32_t lt_mask = lanemask_lt();
    const int64_t warp_id = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    auto position = [&](int64_t k) -> int64_t { return (((k >> 5) * warps + warp_id) << 5) + (k & 31); };
    const bool backface = (flags & DIPL_TRACE_BACKFACE_CULLING) != 0u;
    int64_t next = 0;   // rays this warp has taken (warp-uniform)
    int64_t my = -1;    // this lane's ray, -1 when idle
    QRay r{};
    WtRay w{};
    float tmax = 0.0f, best_t = 0.0f, best_u = 0.0f, best_v = 0.0f;
    int best_prim = -1;
    bool found = false, bad = false;
    // The lane's work: a node (cur >= 0), kQIdle, or a leaf (cur < 0) that waits for `leaf` to be taken; `leaf`: the
    // leaf range whose triangles are tested next, 0 for none.
    int cur = kQIdle, leaf = 0;
    uint32_t steps = 0;
    QStack<STACK> st;
    st.column = sh_stack + threadIdx.x;

    auto start_ray = [&](int64_t cand) {
        my = order ? (int64_t)__ldg(order + cand) : cand;  // the ray's own index (hits go there)
        const bool live = quad_load_ray(rays, my, r, tmax);
        if (LEAF == DIPL_LEAF_WATERTIGHT) w = wt_setup(r.d);
        best_t = tmax, best_u = 0.0f, best_v = 0.0f, best_prim = -1, found = false;
        cur = live && num_nodes >= 0 ? root : kQIdle;
        leaf = 0;
        if (cur < 0) leaf = cur, cur = kQIdle;  // the root is a leaf
        st.sp = 0;
        steps = 0;
    };
    // Pops until a node comes up, the leaf slot and cur both hold a leaf, or the stack is down to `bot`.
    auto advance = [&](int bot) {
        for (;;) {
            if (cur == kQPop) {
                if (st.sp <= bot) {
                    cur = kQIdle;
                    return;
                }
                cur = st.pop();
            }
            if (cur >= 0 || leaf != 0) return;
            leaf = cur;
            cur = kQPop;
        }
    };
    auto give_up = [&]() {  // only a corrupted tree or a step limit gets here
        bad = true;
        cur = kQIdle;
        leaf = 0;
    };
    auto node_step = [&](float lim, int bot) {
        if (++steps > step_limit || cur >= num_nodes || st.sp + 3 > STACK) {
            give_up();
            return;
        }
        float key[4];
        int ref[4];
        quad_children(quads, cur, r, lim, key, ref);
        cur = kQPop;
        if (key[0] < kQMiss) {
            if (st.sp + 3 <= kQShort) {
                if (key[3] < kQMiss) st.push_short(ref[3]);
                if (key[2] < kQMiss) st.push_short(ref[2]);
                if (key[1] < kQMiss) st.push_short(ref[1]);
            } else {
                if (key[3] < kQMiss) st.push(ref[3]);
                if (key[2] < kQMiss) st.push(ref[2]);
                if (key[1] < kQMiss) st.push(ref[1]);
            }
            cur = ref[0];
        }
        advance(bot);
    };
    auto leaf_step = [&](int bot) {
        if (++steps > step_limit) {
            give_up();
            return;
        }
        const int first = leaf_first(leaf), cnt = leaf_count(leaf);
        if (cnt > 0) {  // an unused child slot has no triangles
            float4 p0, p1, p2;
            load_leaf_triangle(tris, first, p0, p1, p2);
            const int prim = __float_as_int(p0.w);
            const float3 a = make_float3(p0.x, p0.y, p0.z), b = make_float3(p1.x, p1.y, p1.z),
                         c = make_float3(p2.x, p2.y, p2.z);
            float b1 = 0.0f, b2 = 0.0f;
            const float t = LEAF == DIPL_LEAF_REF_MT ? mt_ref(a, b, c, r.o, r.d, backface, b1, b2)
                                                     : wt_test(a, b, c, r.o, w, backface, b1, b2);
            // t == kInfinity is the tests' miss value (also when tmax is +inf)
            if (ANY) {
                if (t > r.tmin && t < best_t && t < kInfinity) found = true;
            } else if (t > r.tmin && t < kInfinity && (t < best_t || (t == best_t && found && prim < best_prim))) {
                best_t = t, best_u = b1, best_v = b2, best_prim = prim, found = true;
            }
        }
        if (ANY && found) {
            cur = kQIdle;
            leaf = 0;
        } else if (cnt > 1) {
            leaf = make_leaf_ref(first + 1, cnt - 1);
        } else {
            leaf = 0;
            if (cur < 0) {
                leaf = cur;
                cur = kQPop;
                advance(bot);
            }
        }
    };
    // One step of the warp (called by all lanes; `on`: this lane has work): a node for every lane that has one, then,
    // once kLeafTurn lanes hold a leaf or no lane has a node left, a triangle for every lane that holds a leaf. True
    // when triangles were tested.
    auto warp_step = [&](bool on, float lim, int bot) {
        if (on && cur >= 0 && cur != kQIdle) node_step(lim, bot);
        const uint32_t holds = __ballot_sync(full, on && leaf != 0);
        const uint32_t nodes = __ballot_sync(full, on && cur >= 0 && cur != kQIdle);
        if (holds == 0u || (nodes != 0u && __popc(holds) < kLeafTurn)) return false;
        if (on && leaf != 0) leaf_step(bot);
        return true;
    };
    auto write_hit = [&](int64_t i, float t, float u, float v, int prim) {
        reinterpret_cast<int4*>(hits)[i] =
            prim >= 0 ? make_int4(prim, __float_as_int(t), __float_as_int(u), __float_as_int(v))
                      : make_int4(-1, 0x7F800000, 0, 0);
    };

    // ---- every lane its own ray --------------------------------------------------------------------------------
    if (!PERSIST) {
        const int64_t cand = warp_id * group + lane;
        if (lane < group && cand < n) start_ray(cand);
    }
    for (;;) {
        bool more = false;
        if (PERSIST) {
            const uint32_t idle = __ballot_sync(full, my < 0);
            more = position(next) < n;
            if (more && __popc(idle) >= kRefillLanes) {
                if (my < 0) {
                    const int64_t cand = position(next + __popc(idle & lt_mask));
                    if (cand < n) start_ray(cand);
                }
                next += __popc(idle);
                more = position(next) < n;
            }
        }
        const uint32_t active = __ballot_sync(full, my >= 0);
        if (!more && __popc(active) <= kShareLanes) break;
        warp_step(my >= 0, prune_limit(best_t), 0);
        if (my >= 0 && cur == kQIdle && leaf == 0) {
            if (ANY) occluded[my] = found ? 1 : 0;
            else write_hit(my, best_t, best_u, best_v, found ? best_prim : -1);
            my = -1;
        }
    }

    // ---- the warp's last rays, shared by its lanes -----------------------------------------------------------------
    // A lane without work takes the bottom stack entry (the largest pending subtree) of a lane that has one, with that
    // lane's ray. Lanes prune by the least t any lane has found for the ray (s_lim) but accept hits against their own,
    // so that the smallest (t, primitive id) of all lanes is the record a single lane would produce; each lane that
    // runs out of work merges its best into s_best, and the last one writes the record. Entries leave a stack at the
    // bottom (bot) only while they are in shared memory.
    int owner = lane, bot = 0;
    bool working = my >= 0;
    if (working) {
        s_ray[threadIdx.x] = my;
        s_lanes[threadIdx.x] = 1;
        s_lim[threadIdx.x] = ANY ? 1u : ordered_bits(best_t);
        if (!ANY) {
            s_tmax[threadIdx.x] = tmax;
            s_best[threadIdx.x] = found ? make_float4(best_t, best_u, best_v, __int_as_float(best_prim))
                                        : make_float4(__int_as_float(0x7F800000), 0.0f, 0.0f, __int_as_float(-1));
        }
    }
    for (;;) {
        __syncwarp();  // the last step's shared-memory writes, before other lanes read them
        const uint32_t idle = __ballot_sync(full, !working);
        if (idle == full) break;
        const bool can_give = working && st.sp > bot && bot < kQShort;
        const uint32_t givers = __ballot_sync(full, can_give);
        if (idle && givers) {
            const int rank = __popc(idle & lt_mask);
            const bool take = !working && rank < __popc(givers);
            const int src = take ? nth_set_bit(givers, rank) : lane;
            const int sbot = __shfl_sync(full, bot, src), sowner = __shfl_sync(full, owner, src);
            QRay q;
            q.o.x = __shfl_sync(full, r.o.x, src), q.o.y = __shfl_sync(full, r.o.y, src);
            q.o.z = __shfl_sync(full, r.o.z, src), q.d.x = __shfl_sync(full, r.d.x, src);
            q.d.y = __shfl_sync(full, r.d.y, src), q.d.z = __shfl_sync(full, r.d.z, src);
            q.inv.x = __shfl_sync(full, r.inv.x, src), q.inv.y = __shfl_sync(full, r.inv.y, src);
            q.inv.z = __shfl_sync(full, r.inv.z, src), q.tmin = __shfl_sync(full, r.tmin, src);
            const uint32_t ssteps = __shfl_sync(full, steps, src);
            const float stmax = ANY ? __shfl_sync(full, best_t, src) : 0.0f;
            if (take) {
                owner = sowner;
                r = q;
                if (LEAF == DIPL_LEAF_WATERTIGHT) w = wt_setup(r.d);
                best_t = ANY ? stmax : s_tmax[wbase + owner];
                best_prim = -1, found = false;
                cur = sh_stack[sbot * kTraceThreads + wbase + src], leaf = 0;
                if (cur < 0) leaf = cur, cur = kQIdle;
                steps = ssteps;
                st.sp = bot = 0;
                working = true;
                atomicAdd(&s_lanes[wbase + owner], 1);
            }
            __syncwarp();  // entries read, before their lanes overwrite them
            if (can_give && __popc(givers & lt_mask) < __popc(idle)) {
                ++bot;
                if (bot == st.sp) bot = st.sp = 0;
            }
        }
        const unsigned lb = working ? s_lim[wbase + owner] : 0u;
        if (ANY && working && lb == 0u) cur = kQIdle, leaf = 0;
        const float before = best_t;
        if (warp_step(working, prune_limit(ANY ? best_t : from_ordered_bits(lb)), bot) && working) {
            if (ANY) {
                if (found) s_lim[wbase + owner] = 0u;
            } else if (best_t < before) {
                atomicMin(&s_lim[wbase + owner], ordered_bits(best_t));
            }
        }
        uint32_t done = __ballot_sync(full, working && cur == kQIdle && leaf == 0);
        while (done) {  // one lane at a time: several may have worked on one ray
            if (lane == __ffs(done) - 1) {
                const int o = wbase + owner;
                if (!ANY && found) {
                    const float4 b = s_best[o];
                    if (best_t < b.x || (best_t == b.x && (unsigned)best_prim < (unsigned)__float_as_int(b.w)))
                        s_best[o] = make_float4(best_t, best_u, best_v, __int_as_float(best_prim));
                }
                const int left = s_lanes[o] - 1;
                s_lanes[o] = left;
                if (left == 0) {
                    if (ANY) {
                        occluded[s_ray[o]] = s_lim[o] == 0u ? 1 : 0;
                    } else {
                        const float4 b = s_best[o];
                        write_hit(s_ray[o], b.x, b.y, b.z, __float_as_int(b.w));
                    }
                }
                working = false;
            }
            done &= done - 1u;
            __syncwarp();
        }
    }
    if (bad) atomicOr(err, kErrStack);
}

// ---- ray order ----------------------------------------------------------------------------------------
// On request, batches of at least kReorderMinRays rays are traced in the order of a 30-bit key: the direction's octant
// above a 9-bit-per-axis Morton code of the origin within the batch's origin bounds. A warp's 32 rays then
// start in one small region and head the same way, so its lanes fetch the same nodes and branch alike.
// Records still go to each ray's own index; only the order of work changes, never a result.
constexpr int kReorderBits = 30;

__global__ void __launch_bounds__(256) ray_bounds_kernel(const dipl_ray* __restrict__ rays, int64_t n,
                                                         int* __restrict__ box) {
    float lo[3] = {__int_as_float(0x7F800000), __int_as_float(0x7F800000), __int_as_float(0x7F800000)};
    float hi[3] = {__int_as_float(0xFF800000), __int_as_float(0xFF800000), __int_as_float(0xFF800000)};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 o = __ldg(reinterpret_cast<const float4*>(rays) + 2 * i);
        const float v[3] = {o.x, o.y, o.z};
        for (int a = 0; a < 3; ++a)
            if (isfinite(v[a])) lo[a] = fminf(lo[a], v[a]), hi[a] = fmaxf(hi[a], v[a]);
    }
    for (int a = 0; a < 3; ++a) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(box + a, float_to_ordered(lo[a]));
            atomicMax(box + 3 + a, float_to_ordered(hi[a]));
        }
    }
}

__global__ void ray_box_init_kernel(int* box) {
    if (threadIdx.x < 6)
        box[threadIdx.x] = float_to_ordered(__int_as_float(threadIdx.x < 3 ? 0x7F800000 : 0xFF800000));
}

__device__ __forceinline__ uint32_t spread3_9(uint32_t x) {  // 9 bits to every third bit
    x &= 0x1FFu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

__global__ void __launch_bounds__(256) ray_keys_kernel(const dipl_ray* __restrict__ rays, int64_t n,
                                                       const int* __restrict__ box, uint32_t* __restrict__ keys) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 o = __ldg(reinterpret_cast<const float4*>(rays) + 2 * i);
    const float4 d = __ldg(reinterpret_cast<const float4*>(rays) + 2 * i + 1);
    const float v[3] = {o.x, o.y, o.z};
    uint32_t cell[3];
    for (int a = 0; a < 3; ++a) {
        const float lo = ordered_to_float(__ldg(box + a)), hi = ordered_to_float(__ldg(box + 3 + a));
        const float ext = hi - lo;
        const float q = ext > 0.0f ? (v[a] - lo) * (512.0f / ext) : 0.0f;
        cell[a] = (uint32_t)fminf(fmaxf(q, 0.0f), 511.0f);  // NaN -> 0
    }
    const uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    keys[i] = (oct << 27) | (spread3_9(cell[0]) << 2) | (spread3_9(cell[1]) << 1) | spread3_9(cell[2]);
}

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

template <int LEAF, int STACK, int SHORT>
dipl_status launch_trace(const dipl_bvh* b, const dipl_ray* rays, int64_t n, dipl_hit* hits, uint32_t flags,
                         unsigned long long* counters, cudaStream_t s) {
    auto kernel = trace_kernel<LEAF, STACK, SHORT>;
    // Rays in the coherent order get one lane each (a grid over the whole batch, blocks launched in order): the
    // GPU then works through the sorted order as one moving window and the lanes of a warp start neighbouring rays
    // together; long rays still move to tail_kernel. Measured on the pre-split 16M soup with 16M sorted rays: 137.7
    // ms (Morton30 126.7 ms) against 160.7 ms (147.8 ms) with persistent warps refilling lanes. Rays in the given
    // order keep the persistent grid, where a lane takes its warp's next ray when its own ends (the 1M sphere's
    // grazing rays would otherwise hold their warps).
    const int max_grid = reorder_rays(n, flags) ? std::numeric_limits<int>::max() : persistent_grid<trace_kernel<LEAF, STACK, SHORT>>();
    const int64_t warps_needed = (n + 31) / 32;
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(max_grid, (warps_needed * 32 + kTraceThreads - 1) /
                                                                               kTraceThreads));
    const int num_nodes = b->num_triangles == 0 ? -1 : (int)b->node_capacity;
    if ((reinterpret_cast<uintptr_t>(b->nodes) & 63) != 0) {
        set_last_error("trace: node array is not 64-byte aligned");
        return DIPL_ERR_INTERNAL;
    }
    // a ray takes at most one step per inner node and one per leaf triangle
    const uint32_t steps_cap = trace_step_limit() ? trace_step_limit()
                                                  : (uint32_t)std::min<int64_t>(0xFFFFFFFFll, 2ll * std::max(num_nodes, 0) +
                                                                                                b->num_refs + 64);
    TailQueue tq{nullptr, nullptr, 0, kTailHeaderInts + 2 * STACK, n >= kTailMinRays ? kTailSteps : 0, kTailLanes,
                 steps_cap};
    void* tail_mem = nullptr;
    if (tq.min_steps > 0) {
        const size_t slot_bytes = sizeof(int) * (size_t)tq.slot_ints;
        tq.cap = (int)std::max<int64_t>(1, std::min<int64_t>(n, (int64_t)(kTailBytes / slot_bytes)));
        const size_t bytes = (size_t)tq.cap * slot_bytes;
        dipl_status st = device_alloc(&tail_mem, bytes + 16, s);
        if (st != DIPL_OK) return st;
        tq.slots = static_cast<int*>(tail_mem);
        tq.count = reinterpret_cast<unsigned*>(static_cast<char*>(tail_mem) + bytes);
        const cudaError_t e = cudaMemsetAsync(tq.count, 0, 2 * sizeof(unsigned), s);
        if (e != cudaSuccess) {
            device_free(tail_mem, s);
            return cuda_status(e, "cudaMemsetAsync");
        }
    }
    RayOrder ro;
    if (reorder_rays(n, flags)) {
        dipl_status st = make_ray_order(rays, n, b->d_err, s, ro);
        if (st != DIPL_OK) {
            if (ro.mem) device_free(ro.mem, s);
            device_free(tail_mem, s);
            return st;
        }
    }
    kernel<<<(unsigned)grid, kTraceThreads, 0, s>>>(static_cast<const BNode*>(b->nodes), b->tris, b->root, num_nodes,
                                                   rays, n, hits, flags, counters, b->d_err, tq, ro.order);
    note_launches();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && tq.min_steps > 0) {
        auto tk = tail_kernel<LEAF, STACK>;
        tk<<<(unsigned)persistent_grid<tail_kernel<LEAF, STACK>>(), kTraceThreads, 0, s>>>(static_cast<const BNode*>(b->nodes), b->tris,
                                                                   num_nodes, rays, hits, flags, counters,
                                                                   b->d_err, tq);
        note_launches();
        e = cudaGetLastError();
    }
    device_free(tail_mem, s);
    if (ro.mem) device_free(ro.mem, s);
    DIPL_CUDA(e);
    return DIPL_OK;
}

template <int LEAF, bool ANY, int STACK>
dipl_status launch_quad(const dipl_bvh* b, const dipl_ray* rays, int64_t n, dipl_hit* hits, uint8_t* occ,
                        uint32_t flags, cudaStream_t s) {
    const int num_nodes = b->num_triangles == 0 ? -1 : (int)b->node_capacity;
    // a ray takes at most one step per node and one per leaf triangle
    const uint32_t steps_cap = trace_step_limit() ? trace_step_limit()
                                                  : (uint32_t)std::min<int64_t>(0xFFFFFFFFll, 2ll * std::max(num_nodes, 0) +
                                                                                                  b->num_refs + 64);
    RayOrder ro;
    if (reorder_rays(n, flags)) {
        dipl_status st = make_ray_order(rays, n, b->d_err, s, ro);
        if (st != DIPL_OK) {
            if (ro.mem) device_free(ro.mem, s);
            return st;
        }
    }
    // Batches that the resident lanes hold at once are spread over all warps, down to one ray per warp, whose other
    // lanes then share it (4096 rays of a small frame: 28 us, 60 with 32 rays per warp). Larger ones in the given order
    // run on resident warps that refill idle lanes, since their rays may differ most in length (1M sphere, 4M rays
    // 0.38 ms against 1.11 with one ray per lane; 1M occlusion rays 1.17 against 1.69; where all rays are alike one
    // ray per lane is a little faster: 1M primary rays 0.41 against 0.36). Sorted rays get one lane each: a warp's
    // rays are then of similar length and start together (4M-triangle soup 11.2 against 13.8 ms).
    const int64_t warps = (int64_t)persistent_grid<quad_trace_kernel<LEAF, ANY, false, STACK>>() * (kTraceThreads / 32);
    if (!ro.order && n > warps * 32) {
        const int grid = persistent_grid<quad_trace_kernel<LEAF, ANY, true, STACK>>();
        quad_trace_kernel<LEAF, ANY, true, STACK><<<(unsigned)grid, kTraceThreads, 0, s>>>(
            b->quads, b->tris, b->root, num_nodes, rays, n, hits, occ, flags, b->d_err, steps_cap, 32, nullptr);
    } else {
        const int group = (int)std::min<int64_t>(32, std::max<int64_t>(1, (n + warps - 1) / warps));
        const int64_t per_block = (int64_t)group * (kTraceThreads / 32);
        quad_trace_kernel<LEAF, ANY, false, STACK><<<(unsigned)((n + per_block - 1) / per_block), kTraceThreads, 0, s>>>(
            b->quads, b->tris, b->root, num_nodes, rays, n, hits, occ, flags, b->d_err, steps_cap, group, ro.order);
    }
    note_launches();
    const cudaError_t e = cudaGetLastError();
    if (ro.mem) device_free(ro.mem, s);
    DIPL_CUDA(e);
    return DIPL_OK;
}

template <int LEAF, bool ANY>
dipl_status launch_quad_stack(const dipl_bvh* b, const dipl_ray* rays, int64_t n, dipl_hit* hits, uint8_t* occ,
                              uint32_t flags, cudaStream_t s) {
    // at most 3 entries are pushed per two binary levels
    const int need = 3 * ((b->depth + 1) / 2) + 3;
    if (need <= 64) return launch_quad<LEAF, ANY, 64>(b, rays, n, hits, occ, flags, s);
    if (need <= 160) return launch_quad<LEAF, ANY, 160>(b, rays, n, hits, occ, flags, s);
    return launch_quad<LEAF, ANY, 776>(b, rays, n, hits, occ, flags, s);
}

template <int LEAF>
dipl_status launch_trace_stack(const dipl_bvh* b, const dipl_ray* rays, int64_t n, dipl_hit* hits, uint32_t flags,
                               unsigned long long* counters, cudaStream_t s) {
    // The top 16 stack entries live in shared memory (16 KB per 128-thread block), the rest in local memory.
    // Measured with the one-triangle step (pre-split 16M soup, EMC60 / Morton30, 16M rays; 1M sphere, 4M rays):
    // coherent order 137.8 -> 127.2 ms / 126.7 -> 116.6 ms, given order 212.9 -> 216.2 ms / 159.8 -> 140.4 ms,
    // sphere 0.545 -> 0.501 ms; 8 entries in shared memory gained nothing.
    if (b->depth < 64) return launch_trace<LEAF, 64, 16>(b, rays, n, hits, flags, counters, s);
    if (b->depth < 128) return launch_trace<LEAF, 128, 16>(b, rays, n, hits, flags, counters, s);
    return launch_trace<LEAF, 512, 16>(b, rays, n, hits, flags, counters, s);
}

}  // namespace

dipl_status make_ray_order(const dipl_ray* rays, int64_t n, uint32_t* d_err, cudaStream_t s, RayOrder& ro) {
    const size_t sort_bytes = radix_sort_scratch_bytes(n, 0, kReorderBits, 8);
    const size_t key_bytes = sizeof(uint32_t) * (size_t)n;
    const size_t bytes = 256 + 5 * key_bytes + sort_bytes;
    dipl_status st = device_alloc(&ro.mem, bytes, s);
    if (st != DIPL_OK) return st;
    unsigned char* base = static_cast<unsigned char*>(ro.mem);
    int* box = reinterpret_cast<int*>(base);
    uint32_t* keys = reinterpret_cast<uint32_t*>(base + 256);
    uint32_t* keys_sorted = keys + n;
    uint32_t* keys_alt = keys_sorted + n;
    ro.order = keys_alt + n;
    uint32_t* order_alt = ro.order + n;
    unsigned char* scratch = reinterpret_cast<unsigned char*>(order_alt + n);
    ray_box_init_kernel<<<1, 32, 0, s>>>(box);
    note_launches();
    const int grid = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
    ray_bounds_kernel<<<grid, 256, 0, s>>>(rays, n, box);
    note_launches();
    ray_keys_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(rays, n, box, keys);
    note_launches();
    DIPL_CUDA(cudaGetLastError());
    return radix_sort_pairs(keys, nullptr, keys_sorted, ro.order, keys_alt, order_alt, n, 4, 0, kReorderBits, 8,
                            scratch, s, d_err);
}


dipl_status trace_closest(const dipl_bvh* b, const dipl_ray* rays, int64_t n, dipl_hit* hits, int leaf_test,
                          uint32_t flags, unsigned long long* counters, cudaStream_t s) {
    DIPL_CHECK_ARG(b && n >= 0, "bvh must be non-NULL and n >= 0");
    DIPL_CHECK_ARG(n == 0 || (rays && hits), "rays/hits must be non-NULL");
    DIPL_CHECK_ARG(leaf_test == DIPL_LEAF_REF_MT || leaf_test == DIPL_LEAF_WATERTIGHT, "bad leaf_test");
    DIPL_CHECK_ARG((reinterpret_cast<uintptr_t>(rays) & 15) == 0 && (reinterpret_cast<uintptr_t>(hits) & 15) == 0,
                   "rays and hits must be 16-byte aligned");
    if (n == 0) return DIPL_OK;
    if (b->layout != DIPL_LAYOUT_BINARY || b->bv_type != DIPL_BV_AABB) return trace_closest_ext(b, rays, n, hits, leaf_test, flags, counters, s);
    if (counters)
        return leaf_test == DIPL_LEAF_REF_MT
                   ? launch_trace_stack<DIPL_LEAF_REF_MT>(b, rays, n, hits, flags, counters, s)
                   : launch_trace_stack<DIPL_LEAF_WATERTIGHT>(b, rays, n, hits, flags, counters, s);
    return leaf_test == DIPL_LEAF_REF_MT ? launch_quad_stack<DIPL_LEAF_REF_MT, false>(b, rays, n, hits, nullptr, flags, s)
                                         : launch_quad_stack<DIPL_LEAF_WATERTIGHT, false>(b, rays, n, hits, nullptr, flags, s);
}

dipl_status trace_any(const dipl_bvh* b, const dipl_ray* rays, int64_t n, uint8_t* occ, int leaf_test, uint32_t flags,
                      cudaStream_t s) {
    DIPL_CHECK_ARG(b && n >= 0, "bvh must be non-NULL and n >= 0");
    DIPL_CHECK_ARG(n == 0 || (rays && occ), "rays/occluded must be non-NULL");
    DIPL_CHECK_ARG(leaf_test == DIPL_LEAF_REF_MT || leaf_test == DIPL_LEAF_WATERTIGHT, "bad leaf_test");
    DIPL_CHECK_ARG((reinterpret_cast<uintptr_t>(rays) & 15) == 0, "rays must be 16-byte aligned");
    if (n == 0) return DIPL_OK;
    if (b->layout != DIPL_LAYOUT_BINARY || b->bv_type != DIPL_BV_AABB) return trace_any_ext(b, rays, n, occ, leaf_test, flags, s);
    if (leaf_test == DIPL_LEAF_REF_MT)
        return launch_quad_stack<DIPL_LEAF_REF_MT, true>(b, rays, n, nullptr, occ, flags, s);
    return launch_quad_stack<DIPL_LEAF_WATERTIGHT, true>(b, rays, n, nullptr, occ, flags, s);
}

}  // namespace dipl
