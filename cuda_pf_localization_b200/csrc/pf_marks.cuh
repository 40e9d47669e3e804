// pf_marks.cuh — gated Cartesian log-likelihoods with every landmark rotated once
// per particle.
//
// An observation's residual is the landmark in the particle's frame minus the
// observed vector.  The landmark in the particle's frame (21 of the 29 f32
// operations of a term) is the same for every observation of that landmark, so a
// warp rotates its particles' landmarks once, keeps them on chip and takes the
// observations in their order against them: the operations and the order of
// weight_two, to the bit.
//
// 24 bytes a landmark and lane (two particles) leave room for few warps, so the
// loop lives on independent terms as much as on warps: kMBatch observations at a
// time, the next ones' operands loading meanwhile.  A block has two groups of four
// such warps (markers), a 256-particle tile each: one group's landmarks are in
// tensor memory, whose columns a warp addresses as it likes, the other's in shared
// memory.  Four further warps a group (scouts) predict the next tile's particles
// and form the last one's softmax partial.
//
// 1M particles, 64 landmarks, 256 observations: 188 us against k_weight's 286; the
// f32 pipe is busy 60 % of the time, shared memory 50 %, the issue slots 60 % (the
// 13.3 operations a pair that are left would take 91 us).  With one group (shared
// memory, a warp a scheduler) 284: its latencies show.  One scout a group 217 and,
// at 16 landmarks / 64 observations, 172 against 90 with four: the predict's chain
// is long.  Observations stored twice for packed adds 200 against 190: shared
// memory is the busier unit.  Sorting the observations by landmark instead and
// leaving the terms in shared memory for a second pass: 285 (runs of three or four
// observations behind a rotation leave no independent work).
#pragma once

#include "pf_device.cuh"
#include "umma.cuh"

namespace pfb {
namespace dev {

constexpr int kMObs = 256;      // observations of a call
constexpr int kMMarks = 64;     // landmarks of the table
constexpr int kMUnit = 64;      // particles of a marker warp, two to a lane
constexpr int kMMarkers = 4;    // marker warps of a group
constexpr int kMTile = kMMarkers * kMUnit;
constexpr int kMGroups = 2;     // group 0: tensor memory, group 1: shared memory
constexpr int kMScouts = 4;     // scout warps of a group
constexpr int kMThreads = 32 * kMGroups * (kMMarkers + kMScouts);
constexpr int kMBatch = 4;
constexpr int kMColumns = 8;    // tensor-memory columns of a landmark (six used)
constexpr int kMSlotBytes = 3 * 32 * (int)sizeof(float2);  // shared memory of a landmark
static_assert(kMTile == 2 * kWThreads, "a group takes a softmax tile");
static_assert(kMThreads >= kMObs, "an observation a thread in marks_build");
static_assert(kMMarks * kMColumns == 512, "all columns of tensor memory");

struct MarksSmem {
    // [marker][slot][x, y, z][lane]: landmarks in the frames of the lane's particles
    float2 pred[kMMarkers][kMMarks][3][32];
    float4 rec[kMObs];  // (-ox, -oy, -oz, slot in columns)
    float4 mark_xy[kMMarks];  // (lx, lx, ly, ly)
    float2 mark_z[kMMarks];
    float pose[kMGroups][7][kMTile];
    float ll[kMGroups][2][kMTile];
    uint64_t claimed[kMGroups], ready[kMGroups], taken[kMGroups], scored[kMGroups][2], summed[kMGroups][2];
    int tile[kMGroups];  // of `pose`; negative: no more
    int next;            // tiles of the block claimed so far
    int warp_count[kMThreads / 32];
    int marks, kept;  // landmarks seen, observations kept
    int all_cart;
    int abort;  // a wait has run out
    uint32_t tmem;
};

// Wait of a whole warp for a phase of one of the block's barriers, at most `polls`
// times; false when it or another of the block's waits has run out.
__device__ __forceinline__ bool marks_wait(MarksSmem& sm, uint64_t* bar, int parity,
                                           unsigned polls) {
    const bool ok = __all_sync(~0u, umma::mbar_wait_abort(bar, parity, polls, &sm.abort));
    if (!ok) *const_cast<volatile int*>(&sm.abort) = 1;
    return ok;
}
__device__ __forceinline__ void marks_arrive(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) umma::mbar_arrive(bar);
}

// Observations of ids outside the table are dropped, as in the reference
// (src/cuda/pf_kernels.cu:242); the rest keep their order.
__device__ __forceinline__ void marks_build(MarksSmem& sm, const CObservation* __restrict__ obs,
                                            int nobs, const float* __restrict__ lm, int lm_count) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int* seen = reinterpret_cast<int*>(sm.ll);  // scratch: landmark seen, then its slot
    if (t < kMMarks) seen[t] = 0;
    __syncthreads();
    CObservation o{};
    bool keep = false;
    if (t < nobs) {
        o = obs[t];
        keep = o.id >= 0 && o.id < lm_count;
    }
    if (keep) seen[o.id] = 1;
    const unsigned kept = __ballot_sync(~0u, keep);
    if (lane == 0) sm.warp_count[warp] = __popc(kept);
    const int cart = __syncthreads_and(!keep || o.mode == 0);
    int at = __popc(kept & ((1u << lane) - 1u)), total = 0;
    for (int k = 0; k < kMThreads / 32; ++k) {
        const int c = sm.warp_count[k];
        at += k < warp ? c : 0;
        total += c;
    }
    if (warp == 0) {
        int n = 0;
        for (int i0 = 0; i0 < kMMarks; i0 += 32) {
            const bool on = seen[i0 + lane] != 0;
            const unsigned b = __ballot_sync(~0u, on);
            const int slot = n + __popc(b & ((1u << lane) - 1u));
            n += __popc(b);
            seen[i0 + lane] = slot;
            if (on) {
                const float* l = lm + 3 * (i0 + lane);
                sm.mark_xy[slot] = make_float4(l[0], l[0], l[1], l[1]);
                sm.mark_z[slot] = make_float2(l[2], l[2]);
            }
        }
        if (lane == 0) {
            sm.marks = n;
            sm.kept = total;
            sm.all_cart = cart;
            sm.abort = 0;
            sm.next = kMGroups;
        }
    }
    if (warp == 1 && lane < kMGroups) {
        umma::mbar_init(&sm.claimed[lane], 1);
        umma::mbar_init(&sm.ready[lane], kMScouts);
        umma::mbar_init(&sm.taken[lane], kMMarkers);
        for (int b = 0; b < 2; ++b) {
            umma::mbar_init(&sm.scored[lane][b], kMMarkers);
            umma::mbar_init(&sm.summed[lane][b], 1);
        }
    }
    __syncthreads();
    if (keep) {
        const int slot = seen[o.id];
        sm.rec[at] = make_float4(-o.dx, -o.dy, -o.dz, __int_as_float(slot * kMColumns));
    }
    // the loop takes 2 kMBatch at a time: what it reads past the end is a copy of
    // landmark 0 (its terms are dropped)
    if (t >= total && t < (total + 2 * kMBatch - 1) / (2 * kMBatch) * (2 * kMBatch))
        sm.rec[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();  // the scratch has been read
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ float4 lds4(unsigned a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
template <int kOff>
__device__ __forceinline__ float2 lds2(unsigned a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2 + %3];"
                 : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(kOff));
    return v;
}

// A warp's landmark slots: x, y and z of the lane's two particles.  get() may
// return before the values are there; wait() makes them so.
struct SharedMarks {
    unsigned base;  // shared address of the lane in slot 0
    struct Value {
        float2 x, y, z;
    };
    __device__ __forceinline__ void put(int slot, float2 x, float2 y, float2 z) const {
        const unsigned a = base + slot * kMSlotBytes;
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x.x), "f"(x.y) : "memory");
        asm volatile("st.shared.v2.f32 [%0 + 256], {%1, %2};" ::"r"(a), "f"(y.x), "f"(y.y)
                     : "memory");
        asm volatile("st.shared.v2.f32 [%0 + 512], {%1, %2};" ::"r"(a), "f"(z.x), "f"(z.y)
                     : "memory");
    }
    __device__ __forceinline__ void put_done() const {}
    __device__ __forceinline__ void get(float4 rec, Value& v) const {
        const unsigned a = base + __float_as_uint(rec.w) * (kMSlotBytes / kMColumns);
        v.x = lds2<0>(a);
        v.y = lds2<256>(a);
        v.z = lds2<512>(a);
    }
    template <int kN>
    __device__ __forceinline__ void wait(Value (&)[kN]) const {}
    __device__ __forceinline__ static float2 x(const Value& v) { return v.x; }
    __device__ __forceinline__ static float2 y(const Value& v) { return v.y; }
    __device__ __forceinline__ static float2 z(const Value& v) { return v.z; }
};

struct TensorMarks {
    uint32_t base;  // tensor-memory address of the warp's lanes, column 0
    struct Value {
        float r[8];
    };
    __device__ __forceinline__ void put(int slot, float2 x, float2 y, float2 z) const {
        const float r[8] = {x.x, x.y, y.x, y.y, z.x, z.y, 0.f, 0.f};
        umma::tmem_st8(base + slot * kMColumns, r);
    }
    __device__ __forceinline__ void put_done() const { umma::tmem_wait_st(); }
    __device__ __forceinline__ void get(float4 rec, Value& v) const {
        umma::tmem_ld8(base + __float_as_uint(rec.w), v.r);
    }
    // the values pass through the wait, so no use of them is moved before it
    __device__ __forceinline__ void wait(Value (&v)[4]) const {
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+f"(v[0].r[0]), "+f"(v[0].r[1]), "+f"(v[0].r[2]), "+f"(v[0].r[3]),
                       "+f"(v[0].r[4]), "+f"(v[0].r[5]), "+f"(v[1].r[0]), "+f"(v[1].r[1]),
                       "+f"(v[1].r[2]), "+f"(v[1].r[3]), "+f"(v[1].r[4]), "+f"(v[1].r[5]),
                       "+f"(v[2].r[0]), "+f"(v[2].r[1]), "+f"(v[2].r[2]), "+f"(v[2].r[3]),
                       "+f"(v[2].r[4]), "+f"(v[2].r[5]), "+f"(v[3].r[0]), "+f"(v[3].r[1]),
                       "+f"(v[3].r[2]), "+f"(v[3].r[3]), "+f"(v[3].r[4]), "+f"(v[3].r[5])
                     :
                     : "memory");
    }
    __device__ __forceinline__ static float2 x(const Value& v) {
        return make_float2(v.r[0], v.r[1]);
    }
    __device__ __forceinline__ static float2 y(const Value& v) {
        return make_float2(v.r[2], v.r[3]);
    }
    __device__ __forceinline__ static float2 z(const Value& v) {
        return make_float2(v.r[4], v.r[5]);
    }
};

// The operands of kMBatch observations.
template <typename M>
struct MarksBatch {
    float4 a[kMBatch];
    typename M::Value v[kMBatch];
    __device__ __forceinline__ void load(const M& m, unsigned rec) {
#pragma unroll
        for (int k = 0; k < kMBatch; ++k) {
            a[k] = lds4(rec + 16 * k);
            m.get(a[k], v[k]);
        }
    }
};

enum GateForm { GATE_OFF, GATE_SELECT, GATE_MAX };  // cart_gate_is_max

// The batch's terms added to acc in order; of the last batch only the first n.
template <GateForm kGate, bool kLast, typename M>
__device__ __forceinline__ void marks_add(const MarksBatch<M>& m, const GateConsts& g, float2 ninv,
                                          float2& acc, int n) {
    float2 t[kMBatch];
#pragma unroll
    for (int k = 0; k < kMBatch; ++k) {
        // one word an observation, added twice: a packed add wants it twice in
        // registers, and shared memory is the busier unit
        const float2 x = M::x(m.v[k]), y = M::y(m.v[k]), z = M::z(m.v[k]);
        const float2 ex = make_float2(__fadd_rn(x.x, m.a[k].x), __fadd_rn(x.y, m.a[k].x));
        const float2 ey = make_float2(__fadd_rn(y.x, m.a[k].y), __fadd_rn(y.y, m.a[k].y));
        const float2 ez = make_float2(__fadd_rn(z.x, m.a[k].z), __fadd_rn(z.y, m.a[k].z));
        const float2 r2 = __ffma2_rn(ez, ez, __ffma2_rn(ex, ex, __fmul2_rn(ey, ey)));
        t[k] = __fmul2_rn(r2, ninv);
        if (kGate == GATE_SELECT) {
            t[k].x = r2.x > g.cart_gate2 ? g.cart_out : t[k].x;
            t[k].y = r2.y > g.cart_gate2 ? g.cart_out : t[k].y;
        } else if (kGate == GATE_MAX) {
            t[k].x = max_nan(t[k].x, g.cart_out);
            t[k].y = max_nan(t[k].y, g.cart_out);
        }
    }
#pragma unroll
    for (int k = 0; k < kMBatch; ++k) {
        if (kLast && k >= n) break;
        acc.x = __fadd_rn(acc.x, t[k].x);
        acc.y = __fadd_rn(acc.y, t[k].y);
    }
}

// Log-likelihoods of the lane's two particles against n > 0 observations, the
// landmarks in their slots.
template <GateForm kGate, typename M>
__device__ __forceinline__ float2 marks_sum(const MarksSmem& sm, const M& m, int n,
                                            const GateConsts& g) {
    const float2 ninv = make_float2(-g.inv2rr, -g.inv2rr);
    float2 acc = make_float2(0.f, 0.f);
    unsigned rec = smem_addr(sm.rec);
    MarksBatch<M> p, q;
    p.load(m, rec);
#pragma unroll 1
    for (; n > 2 * kMBatch; n -= 2 * kMBatch) {
        m.wait(p.v);
        q.load(m, rec + 16 * kMBatch);
        marks_add<kGate, false>(p, g, ninv, acc, 0);
        rec += 32 * kMBatch;
        m.wait(q.v);
        p.load(m, rec);
        marks_add<kGate, false>(q, g, ninv, acc, 0);
    }
    m.wait(p.v);
    q.load(m, rec + 16 * kMBatch);
    marks_add<kGate, true>(p, g, ninv, acc, n);
    m.wait(q.v);
    marks_add<kGate, true>(q, g, ninv, acc, n - kMBatch);
    return acc;
}

// The landmarks into the frames of the lane's two particles.
template <typename M>
__device__ __forceinline__ void marks_rotate(const MarksSmem& sm, const PackedPose& k, int marks,
                                             const M& m) {
#pragma unroll 4
    for (int i = 0; i < marks; ++i) {
        const float4 xy = sm.mark_xy[i];
        const float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), k.npx);
        const float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), k.npy);
        const float2 dz = __fadd2_rn(sm.mark_z[i], k.npz);
        const float2 tx = __ffma2_rn(k.k1, dy, __fmul2_rn(k.k2, dz));
        const float2 ty = __ffma2_rn(k.k3, dz, __fmul2_rn(k.k4, dx));
        const float2 tz = __ffma2_rn(k.k5, dx, __fmul2_rn(k.k6, dy));
        const float2 cx = __ffma2_rn(k.m1, ty, __fmul2_rn(k.m2, tz));
        const float2 cy = __ffma2_rn(k.m3, tz, __fmul2_rn(k.m4, tx));
        const float2 cz = __ffma2_rn(k.m5, tx, __fmul2_rn(k.m6, ty));
        m.put(i, __fadd2_rn(__ffma2_rn(k.w2, tx, dx), cx),
              __fadd2_rn(__ffma2_rn(k.w2, ty, dy), cy),
              __fadd2_rn(__ffma2_rn(k.w2, tz, dz), cz));
    }
    m.put_done();
}

// One marker's share of a tile: its landmarks rotated, its log-likelihoods.
template <typename M>
__device__ __forceinline__ float2 marks_unit(const MarksSmem& sm, const M& m, const GateConsts& g,
                                             bool gate_max, const PackedPose& pk) {
    const int n = sm.kept;
    if (n == 0) return make_float2(0.f, 0.f);
    marks_rotate(sm, pk, sm.marks, m);
    if (!(g.gate > 0.0f)) return marks_sum<GATE_OFF>(sm, m, n, g);
    return gate_max ? marks_sum<GATE_MAX>(sm, m, n, g) : marks_sum<GATE_SELECT>(sm, m, n, g);
}

}  // namespace dev
}  // namespace pfb
