// pf_update.cu — prior (reinit), motion update (predict) and landmark
// weighting kernels on the SoA particle planes.
//
// The weighting kernel optionally runs a deferred predict first, so one pass
// over HBM reads the old pose, writes the new pose and the log-likelihood,
// and leaves per-block softmax partials (block max, sum exp(ll - block max)
// in FP64).  The last block to finish combines the partials in block order,
// so M = max ll and S = sum exp(ll - M) are deterministic.
#include <math.h>


#include <algorithm>

#include "pf_device.cuh"
#include "pf_marks.cuh"

namespace pfb {

namespace {

using namespace pfb::dev;
constexpr int kThreads = kBlk;


PlaneSet plane_set(const PfHandle* h) { return {h->planes(0), h->planes(1)}; }

__global__ void __launch_bounds__(kThreads)
    k_reinit(PlaneSet ps, int n, uint64_t seed, uint64_t gen, float3 p0,
             Quat q0, float3 pstd, float3 rstd, CycleCtl* ctl) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const Planes s = pick_planes(ps, ctl->live);
    float nz[6];
    pf_normals6(seed, gen, (uint32_t)i, nz);
    float3 p = make_float3(p0.x + pstd.x * nz[0], p0.y + pstd.y * nz[1],
                           p0.z + pstd.z * nz[2]);
    float3 axis = make_float3(rstd.x * nz[3], rstd.y * nz[4], rstd.z * nz[5]);
    float ang = norm3(axis);
    Quat dq = q_from_axis_angle(axis, ang);
    store_pose(s, i, p, q_product(q0, dq));
}

// Reinitialisation around k planar poses (x, y, yaw) held in device memory:
// particle i starts from pose i mod k at height z with attitude = yaw about
// +z, then the same Gaussian perturbation as k_reinit.
__global__ void __launch_bounds__(kThreads)
    k_reinit_poses(PlaneSet ps, int n, uint64_t seed, uint64_t gen,
                   const float* __restrict__ poses, int k, float z, float3 pstd,
                   float3 rstd, CycleCtl* ctl) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const Planes s = pick_planes(ps, ctl->live);
    const int j = i % k;
    const float x0 = poses[3 * j], y0 = poses[3 * j + 1], yaw = poses[3 * j + 2];
    float sh, ch;
    sincosf(0.5f * yaw, &sh, &ch);
    const Quat q0{ch, 0.0f, 0.0f, sh};
    float nz[6];
    pf_normals6(seed, gen, (uint32_t)i, nz);
    float3 p = make_float3(x0 + pstd.x * nz[0], y0 + pstd.y * nz[1],
                           z + pstd.z * nz[2]);
    float3 axis = make_float3(rstd.x * nz[3], rstd.y * nz[4], rstd.z * nz[5]);
    float ang = norm3(axis);
    Quat dq = q_from_axis_angle(axis, ang);
    store_pose(s, i, p, q_product(q0, dq));
}

__global__ void __launch_bounds__(kThreads)
    k_predict(PlaneSet ps, int n, uint64_t seed, PredictArgs pa,
              CycleCtl* ctl) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const Planes s = pick_planes(ps, ctl->live);
    float3 p;
    Quat q;
    load_pose(s, i, p, q);
    apply_predict(pa, seed, i, p, q);
    store_pose(s, i, p, q);
}

// M and S of the softmax into the control block (weights valid when S is a
// positive finite sum).
__device__ __forceinline__ void softmax_commit(float2 ms, CycleCtl* ctl) {
    const float M = ms.x, S = ms.y;
    ctl->ll_max = M;
    ctl->ll_sumexp = S;
    const int ok = (S > 0.0f && isfinite(S)) ? 1 : 0;
    ctl->weights_valid = ok;
    ctl->wmode = ok ? WMODE_LL : WMODE_UNIFORM;
}

// Softmax partial of one block (two log-likelihoods per thread) + the
// last-block combine into M and S.
__device__ __forceinline__ void softmax_partials(float acc0, bool v0,
                                                 float acc1, bool v1,
                                                 float2* part,
                                                 unsigned* done,
                                                 CycleCtl* ctl) {
    __shared__ bool s_last;
    const float2 pb = block_softmax_partial(acc0, v0, acc1, v1);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = pb;
        __threadfence();
        s_last = (atomicAdd(done, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const float2 ms = softmax_combine(part, gridDim.x);
    if (threadIdx.x == 0) {
        softmax_commit(ms, ctl);
        *done = 0u;
    }
}

// The combine of a sharded filter, once every rank's block partials are in
// part[0, G): one block, the same combine as the last block above, so M and
// S equal the unsharded filter's bit for bit.
__global__ void __launch_bounds__(kWThreads) k_softmax_combine(const float2* part, int G,
                                                              CycleCtl* ctl) {
    const float2 ms = softmax_combine(part, G);
    if (threadIdx.x == 0) softmax_commit(ms, ctl);
}

// Two particles per thread (i and i + kWThreads): every staged observation
// read from shared memory serves both.  Five 128-thread blocks per SM (84
// registers, no spills; 20 warps): measured 1.4 % faster than six (77
// registers) and faster than four, seven or eight.
// kShard: one rank's slice of a sharded filter; block b of the launch is
// block block0 + b of the whole cloud, and the block partials are left for
// the combine that follows the exchange (k_softmax_combine).
template <bool kPredict, bool kShard>
__global__ void __launch_bounds__(kWThreads, 5)
    k_weight(PlaneSet ps, int n, uint64_t seed, PredictArgs pa,
             const CObservation* __restrict__ obs, int nobs,
             const float* __restrict__ lm, int lm_count, float sigma_r,
             float sigma_b, float gate, float* __restrict__ ll,
             float2* part, unsigned* done, CycleCtl* ctl, int arith,
             const CycleArgs* ca, int block0) {
    pdl_wait();
    if (ca) {  // graph replay: this cycle's values
        pa = ca->pa;
        obs = ca->obs;
        nobs = ca->nobs;
    }
    const Planes s = pick_planes(ps, ctl->live);
    const int blk = kShard ? (int)blockIdx.x + block0 : (int)blockIdx.x;
    const int i0 = blk * (2 * kWThreads) + threadIdx.x;
    const int i1 = i0 + kWThreads;
    const bool v0 = i0 < n, v1 = i1 < n;
    float3 p0 = make_float3(0.f, 0.f, 0.f), p1 = p0;
    Quat q0 = {1.f, 0.f, 0.f, 0.f}, q1 = q0;
    if (v0) {
        load_pose(s, i0, p0, q0);
        if (kPredict) {
            apply_predict(pa, seed, i0, p0, q0);
            store_pose(s, i0, p0, q0);
        }
    }
    if (v1) {
        load_pose(s, i1, p1, q1);
        if (kPredict) {
            apply_predict(pa, seed, i1, p1, q1);
            store_pose(s, i1, p1, q1);
        }
    }
    float acc0, acc1;
    const bool cart = weight_two<true>(obs, nobs, lm, lm_count, sigma_r, sigma_b, gate, p0, q0,
                                       p1, q1, arith, acc0, acc1);
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->obs_cart = cart ? 1 : 0;
    if (v0) ll[i0] = acc0;
    if (v1) ll[i1] = acc1;
    if (kShard) {
        const float2 pb = block_softmax_partial(acc0, v0, acc1, v1);
        if (threadIdx.x == 0) part[blk] = pb;
    } else {
        softmax_partials(acc0, v0, acc1, v1, part, done, ctl);
    }
}

// Softmax partial of a 256-particle tile by one warp: block_softmax_partial's
// maximum and its sums, warp by warp of that block, in its order.
__device__ __forceinline__ float2 tile_softmax_partial(const float* s_ll, int count) {
    const int lane = threadIdx.x & 31;
    float a[kWThreads / 32], b[kWThreads / 32];
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWThreads / 32; ++w) {
        const int i0 = 32 * w + lane, i1 = i0 + kWThreads;
        a[w] = i0 < count ? s_ll[i0] : -INFINITY;
        b[w] = i1 < count ? s_ll[i1] : -INFINITY;
        m = fmaxf(m, fmaxf(a[w], b[w]));
    }
    const float bm = warp_max_f(m);
    float sb = 0.0f;
#pragma unroll
    for (int w = 0; w < kWThreads / 32; ++w) {
        const int i0 = 32 * w + lane, i1 = i0 + kWThreads;
        const float e = __fadd_rn(i0 < count ? expf(__fsub_rn(a[w], bm)) : 0.0f,
                                  i1 < count ? expf(__fsub_rn(b[w], bm)) : 0.0f);
        sb = __fadd_rn(sb, warp_sum_f(e));
    }
    return make_float2(bm, sb);
}

// Any observations: k_weight_marks' way with bearings, k_weight's arithmetic by four
// groups of kWThreads threads, a 256-particle tile each at a time.  Sixteen warps an SM
// where k_weight has twenty, and a block's tiles do not divide evenly: 1M x 64 / 256, one
// bearing among them, 389 us against 314, every third one 542 and 469, all of them 846
// and 741 (a particle a thread with scalar arithmetic on half of the block: 2.3 to 2.9
// times k_weight's).
template <bool kPredict>
__device__ __noinline__ void weight_tiles(MarksSmem& sm, const Planes& s, int n, uint64_t seed,
                                          const PredictArgs& pa,
                                          const CObservation* __restrict__ obs, int nobs,
                                          const float* __restrict__ lm, int lm_count,
                                          float sigma_r, float sigma_b, float gate,
                                          float* __restrict__ ll, float2* part) {
    constexpr int kGroups = kMThreads / kWThreads;
    static_assert(sizeof sm.pred >= 5 * kMObs * sizeof(float4), "the staged observations");
    static_assert(sizeof sm.ll >= kGroups * kMTile * sizeof(float), "a tile a group");
    float4* const s_a = reinterpret_cast<float4*>(sm.pred);
    float4 *const s_b = s_a + kMObs, *const s_p = s_b + kMObs;
    const GateConsts g = gate_consts(sigma_r, sigma_b, gate);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = tid / kWThreads, t = tid % kWThreads;
    float* const s_ll = &sm.ll[0][0][0] + group * kMTile;
    auto group_sync = [&]() {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kWThreads) : "memory");
    };
    CObservation o{};
    bool keep = false;
    if (tid < nobs) {
        o = obs[tid];
        keep = o.id >= 0 && o.id < lm_count;
    }
    const unsigned kept = __ballot_sync(~0u, keep);
    int at = __popc(kept & ((1u << lane) - 1u));
    for (int k = 0; k < warp; ++k) at += sm.warp_count[k];  // left by marks_build
    bool is_wild = false;
    if (keep) {
        stage_one(o, lm, at, s_a, s_b, s_p);
        const float4 a = s_a[at];
        is_wild = !tame_landmark(a.x, a.y, a.z);
    }
    // k_weight's chunks: where one starts, whether it has bearings, and wild landmarks
    constexpr int kChunks = kMObs / kObsChunk;
    int start[kChunks + 1] = {0};
    bool mixed[kChunks];
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
        const bool mine = keep && tid / kObsChunk == c;
        start[c + 1] = start[c] + __syncthreads_count(mine);
        mixed[c] = __syncthreads_or(mine && o.mode != 0);
    }
    const bool wild = __syncthreads_or(is_wild);
    for (int tile = blockIdx.x + group * gridDim.x; (long long)tile * kMTile < n;
         tile += kGroups * gridDim.x) {
        const int i0 = tile * kMTile + t;
        float3 p[2];
        Quat q[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + h * kWThreads;
            p[h] = make_float3(0.f, 0.f, 0.f);
            q[h] = {1.f, 0.f, 0.f, 0.f};
            if (i < n) {
                load_pose(s, i, p[h], q[h]);
                if (kPredict) {
                    apply_predict(pa, seed, i, p[h], q[h]);
                    store_pose(s, i, p[h], q[h]);
                }
            }
        }
        const PackedPose pk = pack_pose(p[0], q_conjugate(q[0]), p[1], q_conjugate(q[1]));
        float2 acc = make_float2(0.f, 0.f);
        const bool tame = !wild && tame_pose(pk);
#pragma unroll 1
        for (int c = 0; c < kChunks; ++c) {
            const int at = start[c], cn = start[c + 1] - at;
            if (mixed[c] && !tame)
                scalar_terms(g, p[0], q_conjugate(q[0]), p[1], q_conjugate(q[1]), s_a + at,
                             s_b + at, cn, acc);
            else
                packed_terms(pk, g, s_a + at, s_b + at, s_p + 3 * at, cn, acc);
        }
        if (i0 < n) ll[i0] = acc.x;
        if (i0 + kWThreads < n) ll[i0 + kWThreads] = acc.y;
        s_ll[t] = acc.x;
        s_ll[t + kWThreads] = acc.y;
        group_sync();
        if (t < 32) {
            const float2 pb = tile_softmax_partial(s_ll, min(kMTile, n - tile * kMTile));
            if (t == 0) part[tile] = pb;
        }
        group_sync();
    }
}

// k_weight with every landmark rotated once per particle (pf_marks.cuh), for up to
// kMObs Cartesian observations of up to kMMarks landmarks: one persistent block
// per SM over the same 256-particle tiles, so the log-likelihoods and the softmax
// partials are k_weight's to the bit.  The groups take the block's tiles as they
// finish; the markers predict their first tile themselves, the scouts the others.
// Observations that are not all Cartesian (a device buffer whose contents the host
// has not seen) take weight_tiles.
template <bool kPredict>
__global__ void __launch_bounds__(kMThreads, 1)
    k_weight_marks(PlaneSet ps, int n, uint64_t seed, PredictArgs pa,
                   const CObservation* __restrict__ obs, int nobs, const float* __restrict__ lm,
                   int lm_count, float sigma_r, float sigma_b, float gate,
                   float* __restrict__ ll, float2* part, unsigned* done, CycleCtl* ctl,
                   const CycleArgs* ca, unsigned polls) {
    extern __shared__ __align__(16) unsigned char marks_smem[];
    MarksSmem& sm = *reinterpret_cast<MarksSmem*>(marks_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    if (warp == 0) {
        umma::tmem_alloc(&sm.tmem, kMMarks * kMColumns);
        umma::tmem_relinquish();
    }
    umma::tc_fence_before();
    if (ca) {  // graph replay: this cycle's values
        pa = ca->pa;
        obs = ca->obs;
        nobs = ca->nobs;
    }
    const Planes s = pick_planes(ps, ctl->live);
    marks_build(sm, obs, min(nobs, kMObs), lm, lm_count);  // synchronises
    umma::tc_fence_after();
    const int ntiles = (n + kMTile - 1) / kMTile;
    const bool marker = warp < kMGroups * kMMarkers;
    const int group = marker ? warp / kMMarkers : (warp - kMGroups * kMMarkers) / kMScouts;
    const int w = marker ? warp % kMMarkers : (warp - kMGroups * kMMarkers) % kMScouts;
    bool ok = true;
    if (blockIdx.x == 0 && tid == 0) ctl->obs_cart = sm.all_cart;
    if (!sm.all_cart) {
        weight_tiles<kPredict>(sm, s, n, seed, pa, obs, min(nobs, kMObs), lm, lm_count, sigma_r,
                               sigma_b, gate, ll, part);
    } else if (marker) {
        const GateConsts g = gate_consts(sigma_r, sigma_b, gate);
        const bool gate_max = cart_gate_is_max(g);
        const SharedMarks in_shared{smem_addr(&sm.pred[w][0][0][lane])};
        const TensorMarks in_tensor{sm.tmem + ((uint32_t)(32 * w) << 16)};
        int tile = blockIdx.x + group * gridDim.x;
        for (int k = 0; tile >= 0 && tile < ntiles; ++k) {
            const int l = w * kMUnit + 2 * lane, i = tile * kMTile + l;
            float3 p[2];
            Quat q[2];
            if (k == 0) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    p[h] = make_float3(0.f, 0.f, 0.f);
                    q[h] = {1.f, 0.f, 0.f, 0.f};
                    if (i + h < n) {
                        load_pose(s, i + h, p[h], q[h]);
                        if (kPredict) {
                            apply_predict(pa, seed, i + h, p[h], q[h]);
                            store_pose(s, i + h, p[h], q[h]);
                        }
                    }
                }
            } else {
                auto two = [&](int c) {
                    return *reinterpret_cast<const float2*>(&sm.pose[group][c][l]);
                };
                const float2 x = two(0), y = two(1), z = two(2);
                const float2 qw = two(3), qx = two(4), qy = two(5), qz = two(6);
                marks_arrive(&sm.taken[group]);
                p[0] = make_float3(x.x, y.x, z.x);
                p[1] = make_float3(x.y, y.y, z.y);
                q[0] = {qw.x, qx.x, qy.x, qz.x};
                q[1] = {qw.y, qx.y, qy.y, qz.y};
            }
            const PackedPose pk = pack_pose(p[0], q_conjugate(q[0]), p[1], q_conjugate(q[1]));
            const float2 acc = group == 0 ? marks_unit(sm, in_tensor, g, gate_max, pk)
                                          : marks_unit(sm, in_shared, g, gate_max, pk);
            const int b = k & 1, phase = (k >> 1) & 1;
            if (k > 1 && !marks_wait(sm, &sm.summed[group][b], phase ^ 1, polls)) {
                ok = false;
                break;
            }
            *reinterpret_cast<float2*>(&sm.ll[group][b][l]) = acc;
            if (i + 1 < n)
                *reinterpret_cast<float2*>(&ll[i]) = acc;
            else if (i < n)
                ll[i] = acc.x;
            marks_arrive(&sm.scored[group][b]);
            ok = marks_wait(sm, &sm.ready[group], k & 1, polls);
            if (!ok) break;
            tile = *const_cast<volatile int*>(&sm.tile[group]);
        }
    } else {
        int tile = blockIdx.x + group * gridDim.x;
        for (int k = 0; tile >= 0 && tile < ntiles; ++k) {
            // the group works on tile k; prepare tile k + 1
            if (k > 0 && !(ok = marks_wait(sm, &sm.taken[group], (k - 1) & 1, polls))) break;
            if (w == 0) {
                if (lane == 0) {
                    const int next = atomicAdd(&sm.next, 1) * (int)gridDim.x + blockIdx.x;
                    sm.tile[group] = next < ntiles ? next : -1;
                }
                marks_arrive(&sm.claimed[group]);
            }
            if (!(ok = marks_wait(sm, &sm.claimed[group], k & 1, polls))) break;
            const int next = *const_cast<volatile int*>(&sm.tile[group]);
            for (int l = 32 * w + lane; next >= 0 && l < kMTile; l += 32 * kMScouts) {
                const int i = next * kMTile + l;
                float3 p = make_float3(0.f, 0.f, 0.f);
                Quat q = {1.f, 0.f, 0.f, 0.f};
                if (i < n) {
                    load_pose(s, i, p, q);
                    if (kPredict) {
                        apply_predict(pa, seed, i, p, q);
                        store_pose(s, i, p, q);
                    }
                }
                const float v[7] = {p.x, p.y, p.z, q.w, q.x, q.y, q.z};
#pragma unroll
                for (int c = 0; c < 7; ++c) sm.pose[group][c][l] = v[c];
            }
            marks_arrive(&sm.ready[group]);
            if (w == 0) {
                const int b = k & 1;
                if (!(ok = marks_wait(sm, &sm.scored[group][b], (k >> 1) & 1, polls))) break;
                const float2 pb =
                    tile_softmax_partial(sm.ll[group][b], min(kMTile, n - tile * kMTile));
                if (lane == 0) part[tile] = pb;
                marks_arrive(&sm.summed[group][b]);
            }
            tile = next;
        }
    }
    if (!ok && lane == 0) atomicOr(&ctl->err, ERR_SPIN_TIMEOUT);
    umma::tc_fence_before();
    __threadfence();
    __shared__ bool s_last;
    __syncthreads();
    if (warp == 0) {
        umma::tc_fence_after();
        umma::tmem_dealloc(sm.tmem, kMMarks * kMColumns);
    }
    if (tid == 0) s_last = (atomicAdd(done, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const float2 ms = softmax_combine(part, ntiles);
    if (tid == 0) {
        // after a wait has run out some tiles have the log-likelihoods and partials of
        // another call, whose weights could be anything: the cloud stays uniform
        const bool whole = (__ldcg(&ctl->err) & ERR_SPIN_TIMEOUT) == 0;
        softmax_commit(whole ? ms : make_float2(0.0f, 0.0f), ctl);
        *done = 0u;
    }
}

constexpr int kMarksGrid = 148;

template <bool kPredict>
int launch_marks(PfHandle* h, const PredictArgs& pa, const CObservation* d_obs, int nobs,
                 float sigma_r, float sigma_b, float gate, const CycleArgs* dargs) {
    PFB_CK(cudaFuncSetAttribute(k_weight_marks<kPredict>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(MarksSmem)));
    const int grid = std::min(ceil_div(h->n, 2 * kWThreads), kMarksGrid);
    PFB_CK(launch_pdl(k_weight_marks<kPredict>, grid, kMThreads, sizeof(MarksSmem), h->stream,
                      plane_set(h), h->n, h->seed, pa, d_obs, nobs, h->d_lm, h->lm_count, sigma_r,
                      sigma_b, gate, h->d_ll, reinterpret_cast<float2*>(h->d_part), h->d_done + 0,
                      h->d_ctl, dargs, h->wait_polls));
    return 0;
}

}  // namespace

// Rotating a landmark once saves 21 of an observation's 29 operations for all but
// its first, and costs a block the set-up and two tiles' latency.  k_weight and
// k_weight_marks measured (us, particles x landmarks / observations): 1M x 64/256
// 286 and 188, 1M x 12/128 161 and 100, 1M x 32/96 129 and 104, 1M x 32/64 98 and
// 91, 200k x 32/128 44 and 39, 100k x 64/256 44 and 38, 100k x 64/192 36 and 34,
// 200k x 64/128 44 and 45.
bool weight_by_marks(const PfHandle* h, int nobs, bool cart) {
    return cart && h->weight_variant == 0 && h->lm_count > 0 && h->lm_count <= kMMarks &&
           nobs <= kMObs && nobs >= 96 && nobs >= 2 * h->lm_count &&
           (long long)h->n * (nobs - h->lm_count) >= 16000000;
}

static int weight_arith(const PfHandle* h) {
    return h->weight_variant ? ARITH_SCALAR : h->lm_wild ? ARITH_PACKED_WILD : ARITH_PACKED;
}

int launch_reinit(PfHandle* h, const float p0[3], const float q0[4],
                  const float pstd[3], const float rstd[3]) {
    const int grid = ceil_div(h->n, kThreads);
    KernelScope ks(h, KK_REINIT);
    k_reinit<<<grid, kThreads, 0, h->stream>>>(
        plane_set(h), h->n, h->seed, h->gen, make_float3(p0[0], p0[1], p0[2]),
        Quat{q0[0], q0[1], q0[2], q0[3]},
        make_float3(pstd[0], pstd[1], pstd[2]),
        make_float3(rstd[0], rstd[1], rstd[2]), h->d_ctl);
    PFB_KL();
    return 0;
}

int launch_reinit_poses(PfHandle* h, const float* d_poses, int k, float z,
                        const float pstd[3], const float rstd[3]) {
    const int grid = ceil_div(h->n, kThreads);
    KernelScope ks(h, KK_REINIT);
    k_reinit_poses<<<grid, kThreads, 0, h->stream>>>(
        plane_set(h), h->n, h->seed, h->gen, d_poses, k, z,
        make_float3(pstd[0], pstd[1], pstd[2]),
        make_float3(rstd[0], rstd[1], rstd[2]), h->d_ctl);
    PFB_KL();
    return 0;
}

int launch_predict(PfHandle* h, const PredictArgs& pa) {
    const int grid = ceil_div(h->n, kThreads);
    KernelScope ks(h, KK_PREDICT);
    k_predict<<<grid, kThreads, 0, h->stream>>>(plane_set(h), h->n, h->seed,
                                                pa, h->d_ctl);
    PFB_KL();
    return 0;
}

int launch_weight(PfHandle* h, const PredictArgs& pa, const CObservation* d_obs,
                  int nobs, bool cart, float sigma_r, float sigma_b, float gate,
                  const CycleArgs* dargs) {
    const int grid = ceil_div(h->n, 2 * kWThreads);
    float2* part = reinterpret_cast<float2*>(h->d_part);
    KernelScope ks(h, KK_WEIGHT);
    if (weight_by_marks(h, nobs, cart)) {
        if (pa.enabled ? launch_marks<true>(h, pa, d_obs, nobs, sigma_r, sigma_b, gate, dargs)
                       : launch_marks<false>(h, pa, d_obs, nobs, sigma_r, sigma_b, gate, dargs))
            return -1;
    } else if (pa.enabled) {
        PFB_CK(launch_pdl(k_weight<true, false>, grid, kWThreads, 0, h->stream, plane_set(h),
                          h->n, h->seed, pa, d_obs, nobs, h->d_lm, h->lm_count,
                          sigma_r, sigma_b, gate, h->d_ll, part, h->d_done + 0,
                          h->d_ctl, weight_arith(h), dargs, 0));
    } else {
        PFB_CK(launch_pdl(k_weight<false, false>, grid, kWThreads, 0, h->stream, plane_set(h),
                          h->n, h->seed, pa, d_obs, nobs, h->d_lm, h->lm_count,
                          sigma_r, sigma_b, gate, h->d_ll, part, h->d_done + 0,
                          h->d_ctl, weight_arith(h), dargs, 0));
    }
    PFB_KL();
    h->prefix_valid = false;
    return 0;
}

// One rank's slice of a sharded filter: particles [rank * chunk,
// min((rank + 1) * chunk, n)), predicted and weighted; their block partials
// land at their global block index of d_part (float2 per 256 particles) for
// the exchange.
int launch_weight_shard(PfHandle* h, const PredictArgs& pa, const CObservation* d_obs,
                        int nobs, float sigma_r, float sigma_b, float gate) {
    const long long first = (long long)h->shard_rank * h->shard_chunk;
    const long long last = std::min<long long>(first + h->shard_chunk, h->n);
    if (last <= first) return 0;  // a rank past the end of the cloud
    const int block0 = (int)(first / (2 * kWThreads));
    const int grid = (int)ceil_div_ll(last - first, 2 * kWThreads);
    float2* part = reinterpret_cast<float2*>(h->d_part);
    KernelScope ks(h, KK_WEIGHT);
    PFB_CK(launch_pdl(k_weight<true, true>, grid, kWThreads, 0, h->stream, plane_set(h), h->n,
                      h->seed, pa, d_obs, nobs, h->d_lm, h->lm_count, sigma_r, sigma_b, gate,
                      h->d_ll, part, h->d_done + 0, h->d_ctl,
                      weight_arith(h), (const CycleArgs*)nullptr, block0));
    PFB_KL();
    h->prefix_valid = false;
    return 0;
}

// The softmax of a sharded filter over all ceil(n / 256) block partials.
int launch_softmax_combine(PfHandle* h) {
    const int G = (int)ceil_div_ll(h->n, 2 * kWThreads);
    KernelScope ks(h, KK_WEIGHT);
    k_softmax_combine<<<1, kWThreads, 0, h->stream>>>(
        reinterpret_cast<const float2*>(h->d_part), G, h->d_ctl);
    PFB_KL();
    h->prefix_valid = false;
    return 0;
}

}  // namespace pfb
