// doa_track.cu -- the reference's adaptive tracker on the GPU: per window a
// coarse-to-fine direction search over (l, m), then the beam along the
// estimated direction.
//
// Reference: CpuOptBeamTracker::run_into (src/cpu_opt_beam_tracker.cpp:
// 1619-2454).  Per window (block of K spectra), after the covariance fold
// (doa_cov.cu + launch_doa_fold: smoothing, forward-backward, loading,
// forgetting, loaded Cholesky):
//   level 0   a G x G grid centred on the previous window's estimate (the
//             seeded prior for the first), pitch 2 fov / (G - 1), cells off
//             the unit disk pulled in to r^2 = 0.999 (:806-828); power summed
//             over channels (Bartlett a^H R a, Capon 1 / (a^H (R + eps I)^-1 a),
//             non-finite powers count 0) and its first argmax (:2138-2147);
//   levels    3 x 3 candidates around the running centre at half the previous
//             half-pitch (fov / G halved per level), argmax, then the 3-point
//             quadratic interpolation of the reference on the candidates'
//             centre row and column, applied to the new centre (:2149-2381);
//             with no refinement the interpolation runs on the coarse grid;
//   emission  the window's per-spectrum beam power along the estimate, in the
//             reference's float32 order (the tracker of tracker.cu, mode 0).
// The steering phase is FP64 (k (x l + y m + z n)) reduced to a quadrant, with
// the FP32 Taylor sin / cos of tracker_common.cuh, and powers are FP64 (the
// reference: FP32), so the search follows the reference's geometry and
// decisions and differs only where two candidates' powers tie to float
// precision.  Grid construction, clamping and interpolation are float32 with
// the reference's operation order.
//
// One launch per window, in clusters of one CTA per group of 64 channels.  A
// cluster evaluates 16 coarse points, adds the groups' sums in order through
// distributed shared memory and writes their powers; the cluster that
// finishes last selects the maximum and runs the refinements by itself, its
// CTAs exchanging sums and each selecting alike, so a refinement costs one
// cluster barrier instead of a launch.  A window's matrices do not depend on
// the window before, so its CTAs come up early (programmatic dependent
// launch) and copy their channels' triangles to shared memory while that one
// finishes; the refinements use the same copies.
// What bounds it: the chain of windows and levels.  A level's work is short
// (2e7 FP64 operations for a 16 x 16 grid of 8 elements, 1 us of the FP64
// pipe), its exchanges are latency.
// Measured, 32 windows of 256 spectra, 64 antennas, 8 elements, 16 x 16 grid,
// 2 refinements, the whole call: 1.03 ms, 19 us of it per window (1.35 ms
// with a launch per level, 5.42 ms with a one-thread selection kernel behind
// each).
#include "bf_internal.cuh"
#include "tracker_common.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

namespace bf {
namespace {

constexpr int kMaxM = 16;
constexpr int kMaxGrid = 64;                     // G <= 64: at most 4096 coarse points
constexpr int kMaxPoints = kMaxGrid * kMaxGrid;
constexpr int kChanGroup = 64;                   // channels per partial sum

struct Cd {
    double re, im;
};

// Search state between launches (device memory).
struct SearchState {
    float cl, cm;          // the previous window's estimate: centre of the coarse grid
    unsigned done;         // clusters of the running launch that have written their powers
    unsigned pad[3];
};

struct TrackParams {
    const Cd* S;           // folded covariance [cells][M][M]
    const Cd* Q;           // (S + E I)^-1 [cells][M][M]
    const int* ok;         // [cells]
    const float* pos;      // [A][3]
    const double* kw;      // [F]
    int n_freq, M;
    int capon;
};

__device__ __forceinline__ float2 clamp_disk(float l, float m) {
    const float r2 = __fadd_rn(__fmul_rn(l, l), __fmul_rn(m, m));
    if (r2 > 0.999f) {
        const float s = __fsqrt_rn(__fdiv_rn(0.999f, r2));
        l = __fmul_rn(l, s);
        m = __fmul_rn(m, s);
    }
    return make_float2(l, m);
}

// The reference's 3-point interpolation (src/cpu_opt_beam_tracker.cpp:
// 830-850): an offset only where denom > 0, clamped to [-0.5, 0.5].
__device__ __forceinline__ float interp_offset(float pc, float p_up, float p_down) {
    const float denom = __fadd_rn(__fsub_rn(p_down, __fmul_rn(2.0f, pc)), p_up);
    if (!(denom > 0.0f)) return 0.0f;
    const float d = __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(p_up, p_down)), denom);
    return fminf(0.5f, fmaxf(-0.5f, d));
}

// Cell i of the G x G grid around (cl, cm).
__device__ __forceinline__ float2 coarse_point(int i, float cl, float cm, int G, float fov_l, float fov_m) {
    const float step_l = G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, fov_l), static_cast<float>(G - 1));
    const float step_m = G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, fov_m), static_cast<float>(G - 1));
    const float start_l = __fsub_rn(cl, fov_l), start_m = __fsub_rn(cm, fov_m);
    const int u = i % G, v = i / G;
    return clamp_disk(__fadd_rn(start_l, __fmul_rn(static_cast<float>(u), step_l)),
                      __fadd_rn(start_m, __fmul_rn(static_cast<float>(v), step_m)));
}

constexpr int kCoarseTile = 16;      // coarse points per cluster
constexpr int kFine = 9;             // candidates of a refinement
constexpr int kSearchThreads = kFine * kChanGroup;
constexpr int kMaxGroups = 8;        // CTAs per cluster (a portable cluster)
static_assert(kShardChannels <= kMaxGroups * kChanGroup, "a shard's channels fit one cluster");

struct SearchParams {
    int levels, G;
    float fov_l, fov_m;
    int interp;
    float* dir_out;
};

// First maximum of pw[0, n) by the CTA's threads: strict > over increasing
// index; n when every power is -inf or NaN.  Returned to thread 0.
__device__ __forceinline__ int first_maximum(const float* __restrict pw, int n, float* best_v, int* best_i) {
    const int tid = threadIdx.x;
    float bv = -INFINITY;
    int bi = n;
    for (int i = tid; i < n; i += kSearchThreads) {
        const float x = __ldcg(pw + i);
        if (x > bv) { bv = x; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((tid & 31) == 0) {
        best_v[tid >> 5] = bv;
        best_i[tid >> 5] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kSearchThreads / 32; ++w) {
            if (best_v[w] > bv || (best_v[w] == bv && best_i[w] < bi)) { bv = best_v[w]; bi = best_i[w]; }
        }
    }
    return bi;
}

// The search of window b: the coarse grid by every cluster, the rest by the
// cluster that finishes it.  Sums over channels keep one order at every
// level: within a group channels w, w + 8, ... first, then w = 0 .. 7, then
// the groups.
template <int M>
__global__ void __launch_bounds__(kSearchThreads, 1)
doa_search_kernel(TrackParams p, int b, SearchState* __restrict st, float* __restrict powers, SearchParams q) {
    namespace cg = cooperative_groups;
    constexpr int U = M * (M + 1) / 2;   // upper triangle incl. diagonal
    extern __shared__ Cd xs[];           // [kChanGroup][U]
    __shared__ double kw_s[kChanGroup];
    __shared__ int ok_s[kChanGroup];
    __shared__ double delay_s[kCoarseTile][M];
    __shared__ double red[kChanGroup][kCoarseTile], red_w[8][kCoarseTile];
    __shared__ double part[2][kMaxGroups][kCoarseTile];  // the groups' sums, by level parity
    __shared__ float best_v[kSearchThreads / 32];
    __shared__ int best_i[kSearchThreads / 32];
    __shared__ float fine_pw[kFine];
    __shared__ float centre[4];          // running centre and half-pitches
    __shared__ int s_last;
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, group = static_cast<int>(cluster.block_rank());
    const int n_groups = static_cast<int>(gridDim.y);
    const int f0 = group * kChanGroup, nf = min(kChanGroup, p.n_freq - f0);
    // A CTA's shared memory may be written from another one only once it is
    // known to run: every CTA says so here and waits for the others before the
    // first remote write, with the copies and the coarse sums in between.
    cluster.barrier_arrive();
    // Up to the wait for the window before, a CTA touches only what the fold
    // wrote and the caller's arrays.
    const Cd* X0 = (p.capon ? p.Q : p.S) + (static_cast<size_t>(b) * p.n_freq + f0) * M * M;
    for (int i = tid; i < nf * M * M; i += kSearchThreads) {
        const int c = i / (M * M), e = i % (M * M), r = e / M, k = e % M;
        if (k < r) continue;
        const uint32_t dst =
            static_cast<uint32_t>(__cvta_generic_to_shared(xs + c * U + r * M - r * (r - 1) / 2 + (k - r)));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(X0 + i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (tid < nf) {
        kw_s[tid] = p.kw[f0 + tid];
        ok_s[tid] = p.ok[static_cast<size_t>(b) * p.n_freq + f0 + tid];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // Powers of the group's channels at np points, summed over them into
    // red_w's column sums: thread pt < np returns the group's sum.
    auto point_sum = [&](int np, auto point) -> double {
        for (int i = tid; i < np * M; i += kSearchThreads) {
            const float2 lm = point(i / M);
            // n as direction_from_lm forms it (float), for arrays with z != 0
            const float n = __fsqrt_rn(__fsub_rn(1.0f, __fadd_rn(__fmul_rn(lm.x, lm.x), __fmul_rn(lm.y, lm.y))));
            delay_s[i / M][i % M] = trk::steering_delay(p.pos, i % M, lm.x, lm.y, n);
        }
        __syncthreads();
        const int pt = tid % np, per = kSearchThreads / np;
#pragma unroll 1
        for (int c = tid / np; c < kChanGroup && tid < per * np; c += per) {
            double pw = 0.0;
            if (c < nf) {
                const double k = kw_s[c];
                Cd a[M];
                double mag[M];
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    const float2 w = trk::steering_from_delay(k, delay_s[pt][i]);
                    a[i] = Cd{static_cast<double>(w.x), -static_cast<double>(w.y)};  // exp(-i phase)
                    mag[i] = a[i].re * a[i].re + a[i].im * a[i].im;
                }
                const Cd* X = xs + c * U;
                double diag = 0.0, off = 0.0;
                int t = 0;
#pragma unroll
                for (int r = 0; r < M; ++r) {
                    diag += X[t++].re * mag[r];
                    double tr = 0.0, ti = 0.0;
#pragma unroll
                    for (int e = r + 1; e < M; ++e) {
                        const Cd x = X[t++];
                        tr += x.re * a[e].re - x.im * a[e].im;
                        ti += x.re * a[e].im + x.im * a[e].re;
                    }
                    off += a[r].re * tr + a[r].im * ti;  // Re(conj(a_r) * (X a)_r upper part)
                }
                pw = diag + 2.0 * off;
                if (p.capon) pw = (ok_s[c] && pw > 0.0) ? 1.0 / pw : 0.0;
                if (!isfinite(pw)) pw = 0.0;
            }
            red[c][pt] = pw;
        }
        __syncthreads();
        if (tid < 8 * np) {
            const int w = tid / np;
            double acc = 0.0;
#pragma unroll
            for (int i = 0; i < kChanGroup / 8; ++i) acc += red[w + 8 * i][tid % np];
            red_w[w][tid % np] = acc;
        }
        __syncthreads();
        double s = 0.0;
        if (tid < np) {
#pragma unroll
            for (int w = 0; w < 8; ++w) s += red_w[w][tid];
        }
        return s;
    };
    auto groups_sum = [&](int buf, int pt) {
        double s = 0.0;
        for (int g = 0; g < n_groups; ++g) s += part[buf][g][pt];
        return static_cast<float>(s);  // powers in float, as the reference compares and interpolates them
    };

    // the coarse grid
    const float c0_l = st->cl, c0_m = st->cm;
    const int n_points = q.G * q.G;
    const int i0 = blockIdx.x * kCoarseTile, np = min(kCoarseTile, n_points - i0);
    {
        const double s = point_sum(np, [&](int i) { return coarse_point(i0 + i, c0_l, c0_m, q.G, q.fov_l, q.fov_m); });
        cluster.barrier_wait();
        if (tid < np) *cluster.map_shared_rank(&part[0][group][tid], 0) = s;
    }
    cluster.sync();
    if (group == 0) {
        if (tid < np) {
            powers[i0 + tid] = groups_sum(0, tid);
            __threadfence();
        }
        __syncthreads();
        if (tid == 0) {
            const int last = atomicAdd(&st->done, 1u) + 1 == gridDim.x;
            __threadfence();
            for (int r = 0; r < n_groups; ++r) *cluster.map_shared_rank(&s_last, r) = last;
        }
    }
    cluster.sync();
    if (!s_last) return;

    const float step_l = q.G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, q.fov_l), static_cast<float>(q.G - 1));
    const float step_m = q.G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, q.fov_m), static_cast<float>(q.G - 1));
    {
        // every CTA of the cluster selects for itself, alike
        int bi = first_maximum(powers, n_points, best_v, best_i);
        if (tid == 0) {
            if (bi >= n_points) bi = 0;  // no power above -inf: the first cell, as the reference
            float2 c = coarse_point(bi, c0_l, c0_m, q.G, q.fov_l, q.fov_m);
            if (q.levels == 0 && q.interp) {
                const int u = bi % q.G, v = bi / q.G;
                auto at = [&](int du, int dv) -> float {
                    const int uu = u + du, vv = v + dv;
                    return (uu < 0 || uu >= q.G || vv < 0 || vv >= q.G) ? 0.0f : __ldcg(powers + vv * q.G + uu);
                };
                const float pc = at(0, 0);
                const float du = interp_offset(pc, at(1, 0), at(-1, 0));
                const float dv = interp_offset(pc, at(0, 1), at(0, -1));
                c = clamp_disk(__fadd_rn(c.x, __fmul_rn(du, step_l)), __fadd_rn(c.y, __fmul_rn(dv, step_m)));
            }
            centre[0] = c.x;
            centre[1] = c.y;
            centre[2] = __fmul_rn(__fdiv_rn(q.fov_l, static_cast<float>(q.G)), 0.5f);
            centre[3] = __fmul_rn(__fdiv_rn(q.fov_m, static_cast<float>(q.G)), 0.5f);
        }
        __syncthreads();
    }
    for (int level = 1; level <= q.levels; ++level) {
        const int buf = level & 1;
        auto candidate = [&](int i) {
            const float du = static_cast<float>(i % 3 - 1), dv = static_cast<float>(i / 3 - 1);
            return clamp_disk(__fadd_rn(centre[0], __fmul_rn(du, centre[2])),
                              __fadd_rn(centre[1], __fmul_rn(dv, centre[3])));
        };
        const double s = point_sum(kFine, candidate);
        if (tid < kFine) {
            for (int r = 0; r < n_groups; ++r) *cluster.map_shared_rank(&part[buf][group][tid], r) = s;
        }
        cluster.sync();
        if (tid < kFine) fine_pw[tid] = groups_sum(buf, tid);
        __syncthreads();
        if (tid == 0) {
            float bv = -INFINITY;
            int bi = kFine;
            for (int i = 0; i < kFine; ++i) {
                if (fine_pw[i] > bv) { bv = fine_pw[i]; bi = i; }
            }
            float2 c = candidate(bi >= kFine ? 0 : bi);
            if (q.interp) {
                // the candidates' centre row and column, whichever candidate won
                const float du = interp_offset(fine_pw[4], fine_pw[5], fine_pw[3]);
                const float dv = interp_offset(fine_pw[4], fine_pw[7], fine_pw[1]);
                c = clamp_disk(__fadd_rn(c.x, __fmul_rn(du, centre[2])), __fadd_rn(c.y, __fmul_rn(dv, centre[3])));
            }
            centre[0] = c.x;
            centre[1] = c.y;
            centre[2] = __fmul_rn(centre[2], 0.5f);
            centre[3] = __fmul_rn(centre[3], 0.5f);
        }
        __syncthreads();
    }
    if (group == 0 && tid == 0) {
        // the window's direction (direction_from_lm), centre of the next window's grid
        const float cl = centre[0], cm = centre[1];
        q.dir_out[0] = cl;
        q.dir_out[1] = cm;
        q.dir_out[2] = __fsqrt_rn(__fsub_rn(1.0f, __fadd_rn(__fmul_rn(cl, cl), __fmul_rn(cm, cm))));
        st->cl = cl;
        st->cm = cm;
        st->done = 0;
    }
}

__global__ void doa_track_init_kernel(SearchState* st, float l0, float m0) {
    st->cl = l0;
    st->cm = m0;
    st->done = 0;
}

template <int M>
bf_status launch_search(int m, cudaStream_t stream, const TrackParams& p, int b, SearchState* st, float* powers,
                        int n_groups, const SearchParams& q) {
    if constexpr (M > kMaxM) {
        return set_error(BF_ERR_UNSUPPORTED, "the DOA search supports at most 16 elements after smoothing");
    } else {
        if (m != M) return launch_search<M + 1>(m, stream, p, b, st, powers, n_groups, q);
        const int smem = kChanGroup * M * (M + 1) / 2 * static_cast<int>(sizeof(Cd));
        const cudaError_t err =
            cudaFuncSetAttribute(doa_search_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err != cudaSuccess) return cuda_status(err, "doa_search_kernel smem attribute");
        cudaLaunchAttribute attrs[2] = {};
        attrs[0].id = cudaLaunchAttributeClusterDimension;
        attrs[0].val.clusterDim.x = 1;
        attrs[0].val.clusterDim.y = static_cast<unsigned>(n_groups);
        attrs[0].val.clusterDim.z = 1;
        // each window but the first comes up while the one before it runs: the
        // first waits for the fold, and none of the others starts before it
        attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[1].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>((q.G * q.G + kCoarseTile - 1) / kCoarseTile),
                           static_cast<unsigned>(n_groups));
        cfg.blockDim = dim3(kSearchThreads);
        cfg.dynamicSmemBytes = static_cast<size_t>(smem);
        cfg.stream = stream;
        cfg.attrs = attrs;
        cfg.numAttrs = b > 0 ? 2 : 1;
        return cuda_status(cudaLaunchKernelEx(&cfg, doa_search_kernel<M>, p, b, st, powers, q),
                           "doa_search_kernel launch");
    }
}

uint64_t align256(uint64_t x) { return (x + 255) / 256 * 256; }

}  // namespace

uint64_t doa_track_workspace_bytes(const bf_dims& d, uint64_t block_len, uint64_t subarray) {
    const uint64_t B = d.n_time / block_len, F = d.n_freq, A = d.n_ant;
    const uint64_t M = (subarray > 0 && subarray < A) ? subarray : A;
    return align256(B * F * A * A * 2 * sizeof(int32_t)) + align256(doa_fold_bytes(B * F, M)) +
           align256(kMaxPoints * sizeof(float)) + align256(sizeof(SearchState));
}

bf_status launch_doa_track(cudaStream_t stream, const uint8_t* v, const float* pos, const double* kw,
                           const bf_dims& d, const bf_doa_track_config& c, float* dirs, float* intensity,
                           void* workspace) {
    const uint64_t A = d.n_ant, F = d.n_freq, K = c.block_len;
    const int B = static_cast<int>(d.n_time / K);
    const int M = static_cast<int>((c.subarray > 0 && c.subarray < A) ? c.subarray : A);
    if (M > kMaxM) return set_error(BF_ERR_UNSUPPORTED, "the DOA search supports at most 16 elements after smoothing");
    const uint64_t groups = (F + kChanGroup - 1) / kChanGroup;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    auto* R = reinterpret_cast<int32_t*>(ws);
    ws += align256(static_cast<uint64_t>(B) * F * A * A * 2 * sizeof(int32_t));
    void* fold = ws;
    ws += align256(doa_fold_bytes(static_cast<uint64_t>(B) * F, M));
    auto* powers = reinterpret_cast<float*>(ws);
    ws += align256(kMaxPoints * sizeof(float));
    auto* st = reinterpret_cast<SearchState*>(ws);

    BF_RETURN_IF(launch_doa_covariance(stream, v, R, d, K));
    BF_RETURN_IF(launch_doa_fold(stream, R, d, K, M, c.forgetting, c.diag_load, fold));
    const uint64_t cells = static_cast<uint64_t>(B) * F;
    TrackParams p{};
    p.S = static_cast<const Cd*>(fold);
    p.Q = p.S + cells * M * M;
    p.ok = reinterpret_cast<const int*>(reinterpret_cast<const double*>(p.Q + cells * M * M) + cells);
    p.pos = pos;
    p.kw = kw;
    p.n_freq = static_cast<int>(F);
    p.M = M;
    p.capon = c.estimator != 0;
    doa_track_init_kernel<<<1, 1, 0, stream>>>(st, c.prior_l, c.prior_m);
    BF_RETURN_IF(cuda_status(cudaGetLastError(), "doa_track_init_kernel launch"));
    SearchParams q{};
    q.levels = static_cast<int>(c.levels);
    q.G = static_cast<int>(c.grid);
    q.fov_l = c.fov_l;
    q.fov_m = c.fov_m;
    q.interp = c.interp != 0;
    for (int b = 0; b < B; ++b) {
        q.dir_out = dirs + 3 * b;
        BF_RETURN_IF(launch_search<1>(M, stream, p, b, st, powers, static_cast<int>(groups), q));
    }
    if (intensity == nullptr) return BF_OK;
    // emission: the reference-order tracker along each window's estimate
    return launch_tracker(stream, 0, v, pos, kw, dirs, intensity, nullptr, d, K);
}

}  // namespace bf
