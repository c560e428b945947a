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
// One launch per window and level.  A CTA takes 8 points and a group of 64
// channels (lane = one of 8 points, one of 4 channels), writes one partial
// sum per (point, group), and the CTA that finishes last adds the groups in
// order, takes the argmax and writes the next level's points, or the
// window's direction and the next window's grid.  What bounds it: the chain
// of windows and levels, each a launch whose work (2e7 FP64 operations for a
// 16 x 16 grid of 8 elements, 1 us of the FP64 pipe) is short, so the work is
// spread thin (192 CTAs where 48 left two thirds of the SMs idle) and the
// selection rides in the same launch and in all threads of its CTA.
// A level's matrices do not depend on the level before, so its CTAs come up
// early (programmatic dependent launch) and copy them to shared memory while
// the one before finishes.
// Measured, 32 windows of 256 spectra, 64 antennas, 8 elements, 16 x 16 grid,
// 2 refinements, the whole call: 5.42 ms with a selection kernel of one
// thread behind each level, 1.77 ms with the selection in the same launch,
// 1.35 ms with the matrices copied ahead.
#include "bf_internal.cuh"
#include "tracker_common.cuh"

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
    float cl, cm;          // running centre (l, m)
    float half_l, half_m;  // refinement half-pitch of the current level
    int n_points;          // points of the current level
    unsigned done;         // CTAs of the running level kernel that have written their sums
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

constexpr int kLevelThreads = 256;
constexpr int kPointTile = 8;        // points per CTA
constexpr int kMaxDirect = 256;      // points whose powers fit the fixed shared array

// What a level's selection needs beside the powers.
struct SelectParams {
    int n_groups, level, levels, G;
    float fov_l, fov_m;
    int interp;
    float* dir_out;
    int last_window;
};

// By every thread of the last CTA: the level's powers in float, as the
// reference compares and interpolates them, their first maximum, and the next
// level or window.  pw holds the powers (shared memory).
__device__ __forceinline__ void select_level(const double* __restrict partial, float2* __restrict points,
                                             SearchState* __restrict st, const SelectParams& q, int n,
                                             float* __restrict pw) {
    constexpr int kWarps = kLevelThreads / 32;
    __shared__ float best_v[kWarps];
    __shared__ int best_i[kWarps];
    __shared__ float next[4];  // centre and half-pitches of the next level
    const int tid = threadIdx.x, lane = tid & 31;
    float bv = -INFINITY;
    int bi = n;
    for (int i = tid; i < n; i += kLevelThreads) {
        double s = 0.0;
        for (int g = 0; g < q.n_groups; ++g) s += __ldcg(partial + static_cast<size_t>(g) * kMaxPoints + i);
        const float x = static_cast<float>(s);
        pw[i] = x;
        if (x > bv) { bv = x; bi = i; }  // first maximum: strict > over increasing index
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) {
        best_v[tid >> 5] = bv;
        best_i[tid >> 5] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kWarps; ++w) {
            if (best_v[w] > bv || (best_v[w] == bv && best_i[w] < bi)) { bv = best_v[w]; bi = best_i[w]; }
        }
        if (bi >= n) bi = 0;  // every power NaN-free and -inf: the first cell, as the reference
        const float2 best = points[bi];
        float cl = best.x, cm = best.y, half_l = st->half_l, half_m = st->half_m;
        if (q.level == 0) {
            if (q.levels == 0 && q.interp) {
                const int u = bi % q.G, v = bi / q.G;
                auto at = [&](int du, int dv) -> float {
                    const int uu = u + du, vv = v + dv;
                    return (uu < 0 || uu >= q.G || vv < 0 || vv >= q.G) ? 0.0f : pw[vv * q.G + uu];
                };
                const float pc = pw[bi];
                const float du = interp_offset(pc, at(1, 0), at(-1, 0));
                const float dv = interp_offset(pc, at(0, 1), at(0, -1));
                const float step_l = q.G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, q.fov_l), static_cast<float>(q.G - 1));
                const float step_m = q.G == 1 ? 0.0f : __fdiv_rn(__fmul_rn(2.0f, q.fov_m), static_cast<float>(q.G - 1));
                const float2 c = clamp_disk(__fadd_rn(cl, __fmul_rn(du, step_l)), __fadd_rn(cm, __fmul_rn(dv, step_m)));
                cl = c.x;
                cm = c.y;
            }
            half_l = __fdiv_rn(q.fov_l, static_cast<float>(q.G));
            half_m = __fdiv_rn(q.fov_m, static_cast<float>(q.G));
        } else if (q.interp) {
            // the candidates' centre row and column, whichever candidate won
            const float du = interp_offset(pw[4], pw[5], pw[3]);
            const float dv = interp_offset(pw[4], pw[7], pw[1]);
            const float2 c = clamp_disk(__fadd_rn(cl, __fmul_rn(du, half_l)), __fadd_rn(cm, __fmul_rn(dv, half_m)));
            cl = c.x;
            cm = c.y;
        }
        if (q.level < q.levels) {
            half_l = __fmul_rn(half_l, 0.5f);
            half_m = __fmul_rn(half_m, 0.5f);
        } else {
            // the window's direction (direction_from_lm)
            q.dir_out[0] = cl;
            q.dir_out[1] = cm;
            q.dir_out[2] = __fsqrt_rn(__fsub_rn(1.0f, __fadd_rn(__fmul_rn(cl, cl), __fmul_rn(cm, cm))));
        }
        st->cl = cl;
        st->cm = cm;
        st->half_l = half_l;
        st->half_m = half_m;
        st->n_points = q.level < q.levels ? 9 : q.G * q.G;
        st->done = 0;
        next[0] = cl;
        next[1] = cm;
        next[2] = half_l;
        next[3] = half_m;
    }
    __syncthreads();
    if (q.level < q.levels) {
        if (tid < 9) {
            const float du = static_cast<float>(tid % 3 - 1), dv = static_cast<float>(tid / 3 - 1);
            points[tid] = clamp_disk(__fadd_rn(next[0], __fmul_rn(du, next[2])),
                                     __fadd_rn(next[1], __fmul_rn(dv, next[3])));
        }
    } else if (!q.last_window) {
        for (int i = tid; i < q.G * q.G; i += kLevelThreads) {
            points[i] = coarse_point(i, next[0], next[1], q.G, q.fov_l, q.fov_m);
        }
    }
}

// Bartlett or Capon power of window `b` at the points, summed over each
// 64-channel group (partial[group][point]: channels w, w + 8, ... of the
// group first, then w = 0 .. 7), and the selection by the last CTA.
template <int M>
__global__ void __launch_bounds__(kLevelThreads) doa_level_kernel(TrackParams p, int b, float2* __restrict points,
                                                                  SearchState* __restrict state,
                                                                  double* __restrict partial, SelectParams q) {
    constexpr int U = M * (M + 1) / 2;   // upper triangle incl. diagonal
    extern __shared__ Cd xs[];           // [kChanGroup][U], then the powers of grids above kMaxDirect points
    float* pw_large = reinterpret_cast<float*>(xs + kChanGroup * U);
    __shared__ float pw_small[kMaxDirect];
    __shared__ double red[kChanGroup][kPointTile];
    __shared__ double red_w[8][kPointTile];
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pl = lane & 7, cl = lane >> 3;
    const int pt = blockIdx.x * kPointTile + pl;
    const int group = blockIdx.y;
    // Up to the wait for the level before, a CTA touches only what the fold
    // wrote: the triangles of its warps' eight channels, all loads in flight
    // at once.  Once past it, it lets the next level's CTAs come up.
#pragma unroll 1
    for (int i = 0; i < kChanGroup / 8; ++i) {
        const int c = 4 * warp + (i & 3) + 32 * (i >> 2), f = group * kChanGroup + c;
        if (f >= p.n_freq) continue;
        const Cd* X = (p.capon ? p.Q : p.S) + (static_cast<size_t>(b) * p.n_freq + f) * M * M;
        for (int e = lane; e < M * M; e += 32) {
            const int r = e / M, k = e % M;
            if (k < r) continue;
            const uint32_t dst = static_cast<uint32_t>(
                __cvta_generic_to_shared(xs + c * U + r * M - r * (r - 1) / 2 + (k - r)));
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(X + e) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n_points = state->n_points;
    const float2 lm = pt < n_points ? points[pt] : make_float2(0.f, 0.f);
    const double l = lm.x, m = lm.y;
    // n as direction_from_lm forms it (float), for arrays with z != 0
    const double n = __fsqrt_rn(__fsub_rn(1.0f, __fadd_rn(__fmul_rn(lm.x, lm.x), __fmul_rn(lm.y, lm.y))));
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
#pragma unroll 1
    for (int c = 4 * warp + cl; c < kChanGroup; c += 32) {
        const int f = group * kChanGroup + c;
        double pw = 0.0;
        if (f < p.n_freq && pt < n_points) {
            const size_t cell = static_cast<size_t>(b) * p.n_freq + f;
            const double k = p.kw[f];
            Cd a[M];
            double mag[M];
#pragma unroll
            for (int i = 0; i < M; ++i) {
                const double delay = trk::steering_delay(p.pos, i, l, m, n);
                const float2 w = trk::steering_from_delay(k, delay);
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
            if (p.capon) pw = (p.ok[cell] && pw > 0.0) ? 1.0 / pw : 0.0;
            if (!isfinite(pw)) pw = 0.0;
        }
        red[c][pl] = pw;
    }
    __syncthreads();
    if (threadIdx.x < 8 * kPointTile) {
        const int w = threadIdx.x >> 3;
        double acc = 0.0;
#pragma unroll
        for (int i = 0; i < kChanGroup / 8; ++i) acc += red[w + 8 * i][threadIdx.x & 7];
        red_w[w][threadIdx.x & 7] = acc;
    }
    __syncthreads();
    if (threadIdx.x < kPointTile && blockIdx.x * kPointTile + threadIdx.x < n_points) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red_w[w][threadIdx.x];
        partial[static_cast<size_t>(group) * kMaxPoints + blockIdx.x * kPointTile + threadIdx.x] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&state->done, 1u) + 1 == gridDim.x * gridDim.y;
        __threadfence();
    }
    __syncthreads();
    if (s_last) select_level(partial, points, state, q, n_points, n_points <= kMaxDirect ? pw_small : pw_large);
}

__global__ void doa_track_init_kernel(SearchState* st, float2* points, float l0, float m0, int G, float fov_l,
                                      float fov_m) {
    for (int i = threadIdx.x; i < G * G; i += blockDim.x) points[i] = coarse_point(i, l0, m0, G, fov_l, fov_m);
    if (threadIdx.x == 0) {
        st->n_points = G * G;
        st->done = 0;
    }
}

template <int M>
bf_status launch_level(int m, cudaStream_t stream, const TrackParams& p, int b, float2* points, SearchState* st,
                       double* partial, int n_points, const SelectParams& q) {
    if constexpr (M > kMaxM) {
        return set_error(BF_ERR_UNSUPPORTED, "the DOA search supports at most 16 elements after smoothing");
    } else {
        if (m != M) return launch_level<M + 1>(m, stream, p, b, points, st, partial, n_points, q);
        const dim3 grid(static_cast<unsigned>((n_points + kPointTile - 1) / kPointTile),
                        static_cast<unsigned>(q.n_groups));
        const int smem = kChanGroup * M * (M + 1) / 2 * static_cast<int>(sizeof(Cd)) +
                         (n_points > kMaxDirect ? n_points * static_cast<int>(sizeof(float)) : 0);
        const cudaError_t err =
            cudaFuncSetAttribute(doa_level_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err != cudaSuccess) return cuda_status(err, "doa_level_kernel smem attribute");
        // each level but the first comes up while the one before it runs
        // (programmatic dependent launch): the first waits for the fold, and
        // none of the others starts before it
        cudaLaunchAttribute overlap{};
        overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        overlap.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(kLevelThreads);
        cfg.dynamicSmemBytes = static_cast<size_t>(smem);
        cfg.stream = stream;
        cfg.attrs = &overlap;
        cfg.numAttrs = b > 0 || q.level > 0 ? 1 : 0;
        return cuda_status(cudaLaunchKernelEx(&cfg, doa_level_kernel<M>, p, b, points, st, partial, q),
                           "doa_level_kernel launch");
    }
}

uint64_t align256(uint64_t x) { return (x + 255) / 256 * 256; }

}  // namespace

uint64_t doa_track_workspace_bytes(const bf_dims& d, uint64_t block_len, uint64_t subarray) {
    const uint64_t B = d.n_time / block_len, F = d.n_freq, A = d.n_ant;
    const uint64_t M = (subarray > 0 && subarray < A) ? subarray : A;
    const uint64_t groups = (F + kChanGroup - 1) / kChanGroup;
    return align256(B * F * A * A * 2 * sizeof(int32_t)) + align256(doa_fold_bytes(B * F, M)) +
           align256(kMaxPoints * sizeof(float2)) + align256(groups * kMaxPoints * sizeof(double)) +
           align256(sizeof(SearchState));
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
    auto* points = reinterpret_cast<float2*>(ws);
    ws += align256(kMaxPoints * sizeof(float2));
    auto* partial = reinterpret_cast<double*>(ws);
    ws += align256(groups * kMaxPoints * sizeof(double));
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
    const int G = static_cast<int>(c.grid), L = static_cast<int>(c.levels);
    doa_track_init_kernel<<<1, 256, 0, stream>>>(st, points, c.prior_l, c.prior_m, G, c.fov_l, c.fov_m);
    BF_RETURN_IF(cuda_status(cudaGetLastError(), "doa_track_init_kernel launch"));
    SelectParams q{};
    q.n_groups = static_cast<int>(groups);
    q.levels = L;
    q.G = G;
    q.fov_l = c.fov_l;
    q.fov_m = c.fov_m;
    q.interp = c.interp != 0;
    for (int b = 0; b < B; ++b) {
        q.dir_out = dirs + 3 * b;
        q.last_window = b + 1 == B;
        for (q.level = 0; q.level <= L; ++q.level) {
            BF_RETURN_IF(launch_level<1>(M, stream, p, b, points, st, partial, q.level == 0 ? G * G : 9, q));
        }
    }
    if (intensity == nullptr) return BF_OK;
    // emission: the reference-order tracker along each window's estimate
    return launch_tracker(stream, 0, v, pos, kw, dirs, intensity, nullptr, d, K);
}

}  // namespace bf
