// tracker.cu -- dynamic single-beam tracker (n_beams == 1).
//
// Reference behaviour: beam_tracker_cpu_packed_intensity_into
// (src/beam_tracker.cpp:90-146) computes one weight set per integration
// window from the window's direction (evaluated at the window's first sample,
// src/beam_tracker.cpp:52-76) and writes the per-spectrum power [T][F][1].
// The reference GPU trackers (src/cuda_beam_tracker_v5.cu:137-273) compute
// the same weights on the device in FP64.
//
// mode 0 (this file): reference float32 operation order.  One CTA per
//   (window, 32-channel block); the window's weights are generated once into
//   shared memory ([A][32] float2) with the FP64 delay, FP64 phase and FP64
//   sin/cos rounded to float exactly as src/weights.cpp:42-55.  Each of the 8
//   warps takes two of every 16 spectra of the window (lanes = channels,
//   64-byte coalesced rows) in packed f32x2 pairs; the optional per-window sum
//   is taken in increasing time through a small shared-memory stage, as
//   src/temporal_integration.cpp:95-109 would sum the per-spectrum output.
//   Bound by instruction issue: eight unfused operations per complex
//   multiply-add on the pairs, beside decode and weight loads that two spectra
//   share (8192 spectra of 64 antennas in windows of 256: 116 us, 129 with
//   scalar arithmetic; 16384 in windows of 1024, summed: 338 us, 391).
// mode 1 (tracker_stream.cu): the HBM streaming kernel.
#include "bf_internal.cuh"
#include "packed_f32.cuh"

#include <algorithm>

namespace bf {

bf_status launch_tracker_stream(cudaStream_t stream, const uint8_t* v, const float* pos,
                                const double* k, const float* dirs, float* intensity,
                                float* integrated, const bf_dims& d, uint64_t spectra);

namespace {

constexpr int kSlots = 8;
constexpr int kStep = 2 * kSlots;  // spectra per step of the CTA

__global__ void __launch_bounds__(kSlots * 32)
tracker_exact_kernel(const uint8_t* __restrict__ v, const float* __restrict__ pos,
                     const double* __restrict__ kw, const float* __restrict__ dirs,
                     float* __restrict__ intensity, float* __restrict__ integrated, int n_time,
                     int n_freq, int n_ant, int spectra, float one) {
    extern __shared__ float2 ws[];  // [A][32]
    __shared__ float pw[kStep][32];
    const int win = blockIdx.x;
    const int f0 = blockIdx.y * 32;
    const int lane = threadIdx.x & 31, slot = threadIdx.x >> 5;

    const double dx = dirs[3 * win], dy = dirs[3 * win + 1], dz = dirs[3 * win + 2];
    for (int i = threadIdx.x; i < n_ant * 32; i += blockDim.x) {
        const int a = i >> 5, f = f0 + (i & 31);
        float2 w = make_float2(0.f, 0.f);
        if (f < n_freq) {
            const double delay = __dadd_rn(__dadd_rn(__dmul_rn((double)pos[3 * a], dx),
                                                     __dmul_rn((double)pos[3 * a + 1], dy)),
                                           __dmul_rn((double)pos[3 * a + 2], dz));
            const double phase = __dmul_rn(kw[f], delay);
            double s, c;
            sincos(phase, &s, &c);
            w = make_float2(static_cast<float>(c), static_cast<float>(s));
        }
        ws[i] = w;
    }
    __syncthreads();

    const int f = f0 + lane;
    const int t0 = win * spectra;
    const int t1 = min(t0 + spectra, n_time);
    const uint64_t plus = pack2(one, one), minus = pack2(-one, -one);
    float acc = 0.f;
    for (int tb = t0; tb < t1; tb += kStep) {
        const int t = tb + 2 * slot;
        F2 power{0.f, 0.f};
        if (t < t1 && f < n_freq) {
            const uint8_t* row = v + (static_cast<size_t>(t) * n_freq + f) * n_ant;
            const bool two = t + 1 < t1;
            const uint8_t* next = row + (two ? static_cast<size_t>(n_freq) * n_ant : 0);
            uint64_t sr = 0, si = 0;
            for (int a0 = 0; a0 < n_ant; a0 += 16) {
                const uint4 r0 = __ldg(reinterpret_cast<const uint4*>(row + a0));
                const uint4 r1 = __ldg(reinterpret_cast<const uint4*>(next + a0));
                const uint32_t x0[4] = {r0.x, r0.y, r0.z, r0.w}, x1[4] = {r1.x, r1.y, r1.z, r1.w};
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int bit = 8 * (j & 3);
                    const float2 w = ws[(a0 + j) * 32 + lane];
                    const uint64_t wr = pack2(w.x, w.x), wi = pack2(w.y, w.y);
                    const uint64_t xr = pack2(nibble_float(x0[j >> 2], bit), nibble_float(x1[j >> 2], bit));
                    const uint64_t xi = pack2(nibble_float(x0[j >> 2], bit + 4), nibble_float(x1[j >> 2], bit + 4));
                    sr = add2(sr, fma2(mul2(wi, xi), minus, mul2(wr, xr)));
                    si = add2(si, fma2(mul2(wi, xr), plus, mul2(wr, xi)));
                }
            }
            power = unpack2(fma2(mul2(si, si), plus, mul2(sr, sr)));
            if (intensity != nullptr) {
                intensity[static_cast<size_t>(t) * n_freq + f] = power.x;
                if (two) intensity[static_cast<size_t>(t + 1) * n_freq + f] = power.y;
            }
        }
        if (integrated != nullptr) {
            pw[2 * slot][lane] = power.x;
            pw[2 * slot + 1][lane] = power.y;
            __syncthreads();
            if (slot == 0) {
                for (int s = 0; s < kStep && tb + s < t1; ++s) acc = __fadd_rn(acc, pw[s][lane]);
            }
            __syncthreads();
        }
    }
    if (integrated != nullptr && slot == 0 && f < n_freq) {
        integrated[static_cast<size_t>(win) * n_freq + f] = acc;
    }
}

}  // namespace

bf_status launch_tracker(cudaStream_t stream, int mode, const uint8_t* v, const float* pos,
                         const double* k, const float* dirs, float* intensity, float* integrated,
                         const bf_dims& d, uint64_t spectra) {
    if (mode == 1) {
        return launch_tracker_stream(stream, v, pos, k, dirs, intensity, integrated, d, spectra);
    }
    const uint64_t W = window_count(d.n_time, spectra);
    if (W > 0x7fffffffull || d.n_time > 0x7fffffffull) {
        return set_error(BF_ERR_OVERFLOW, "CUDA tracker grid exceeds the supported size");
    }
    const size_t smem = d.n_ant * 32 * sizeof(float2);
    cudaError_t err = cudaFuncSetAttribute(tracker_exact_kernel,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           static_cast<int>(smem));
    if (err != cudaSuccess) return cuda_status(err, "tracker_exact_kernel smem attribute");
    const dim3 grid(static_cast<unsigned>(W), static_cast<unsigned>((d.n_freq + 31) / 32));
    tracker_exact_kernel<<<grid, kSlots * 32, smem, stream>>>(
        v, pos, k, dirs, intensity, integrated, static_cast<int>(d.n_time),
        static_cast<int>(d.n_freq), static_cast<int>(d.n_ant),
        static_cast<int>(std::min<uint64_t>(spectra, d.n_time)), 1.0f);
    return cuda_status(cudaGetLastError(), "tracker_exact_kernel launch");
}

}  // namespace bf
