// tracker_stream.cu -- HBM streaming tracker kernel (bf_tracker mode 1).
//
// Same product as the reference trackers (src/beam_tracker.cpp:90-146 on the
// CPU, src/cuda_beam_tracker_v5.cu:137-273 on the GPU): one steering weight
// set per integration window, per-spectrum power |sum_a w_a x_a|^2 for a
// single beam, plus (new) the per-window sum.
//
// The kernel reads every voltage byte exactly once with 128-bit loads and is
// meant to run at HBM speed.  At 64 antennas a scalar complex MAC costs about
// 12 ALU instructions per input byte, which would make the kernel ALU-bound,
// so the MAC runs on the tensor pipe instead with the voltage fed straight
// from registers:
//   * Windows above 16 spectra use the integer form of tracker_common.cuh:
//     voltages as int8 (16 x the int4 values, one mask per four components),
//     each weight as four signed base-256 digits of rint(w 2^30), and one
//     mma.m16n8k32 per 16 spectra x 16 antennas whose eight columns are
//     (re, im) x the digits.  Everything before |.|^2 is exact but the last
//     two roundings that put the digit sums together.
//   * Windows of one block use fp16: packed bytes become fp16 pairs with two
//     LOP3s (the nibble placed in the mantissa of 1024.0 with its sign bit
//     flipped) and one half2 subtract / fma, weights an fp16 hi + lo pair, and
//     mma.m16n8k16 multiplies 16 spectra x 8 antennas into (re, im) x (hi, lo),
//     added in fp32.  There the digits would cost more to form than the
//     shorter decode saves.
//   * The weights come from FP64 delay and phase, reduced mod 2*pi in FP64,
//     then float sin/cos.
//   * Lanes (g, q) of the fragment map to spectra g, g+8 and to the q-th
//     quarter of the antenna row, so each thread loads its A/4 contiguous
//     bytes of two rows; the K order of the contraction is permuted to match
//     (only the weights need to follow it).
// A CTA of 8 warps takes 8 consecutive channels (512 contiguous bytes per
// spectrum at 64 antennas), a warp one channel, in blocks of 16 spectra.  The
// FP64 delays of the CTA's windows are formed once and each weight once per
// warp (a lane forms the two antennas of a fragment word), passed to the
// fragment columns through shared memory: forming them per fragment repeated
// each weight four times in half of the lanes.  Two forms:
//   * long windows, one per CTA: two blocks' rows in registers, the next two
//     on their way;
//   * short windows, a run of up to 16 per CTA: each lane fills a ring of
//     kDepth blocks for itself with cp.async and reads it back itself, so the
//     loads run ahead over the window ends without registers or barriers.
// Per-spectrum powers are staged four blocks at a time so that each
// spectrum's 8 channels are written as one 32-byte sector.
// What bounds it: HBM for long windows (131072 spectra in windows of 1024,
// 64 antennas: 0.471 ms = 6.0 TB/s; in the fp16 form issue, 0.637 ms); for
// windows of 10 spectra the weights' arithmetic and the six empty rows of
// each block (15360 spectra, both outputs, 0.252 ms; 0.819 with weights formed
// per fragment and one window per CTA).  Other windows at 64 antennas: 32000
// spectra in windows of 320 0.126 ms (0.189 at first), 8000 in windows of 32
// 0.050 (0.147).  Against 64 bits the window sums of the integer form are off
// by 4-6e-8, those of the fp16 form by 5e-8 (32 antennas) to 4e-7 (256).
#include "bf_internal.cuh"
#include "tracker_common.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace bf {
namespace {

using namespace trk;

constexpr int kChannelsPerCta = 8;
constexpr int kMaxRun = 16;         // windows per CTA
// A run is as many windows as fit in these spectra, one at least: enough for two
// windows of the longest length, whose weights and first loads then overlap the
// window before (with 80, windows of 64 were 3 to 8 % slower, of 16 3 %; with
// 320 none was faster).  Half of kMaxRun made windows of 1 3 % slower at 64
// antennas.
constexpr int kRunSpectra = 160;
constexpr int kWantedCtas = 4 * 4 * 148;
// Longest window of the ring form: in the fp16 form windows of 100 took 75 us
// in it and 77 us in the long form (9999 spectra), windows of 320 179 and 166
// us (32000).
constexpr int kShortWindow = 64;
// Longest window in the fp16 form (one block), here and in the served tracker;
// longer ones take the integer form.
constexpr int kHalfWindow = 16;
constexpr int kStageBlocks = 4;     // blocks of per-spectrum powers between barriers

// Blocks of 16 spectra in a warp's ring (1 KB each at 64 antennas).
template <int A>
__host__ __device__ constexpr int ring_depth() { return A == 32 ? 8 : A == 64 ? 4 : A == 128 ? 3 : 2; }

// Bytes of a warp's weights: fp16 parts, or digit rows.
template <int A, bool kInt8>
__host__ __device__ constexpr int part_bytes() { return kInt8 ? kDigitRows * A : 8 * A; }

template <int N>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src, bool on) {
    // a source size of 0 reads nothing and zero-fills
    if constexpr (N == 8) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(on ? 8 : 0) : "memory");
    } else {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16 : 0)
                     : "memory");
    }
}

// Blocks of a run of windows in order: 16 spectra at a time, a window's last
// block as short as the window leaves it.
struct BlockCursor {
    int win, t, end;  // window, first spectrum of the block, end of the window
    __device__ __forceinline__ void start(int w, int spectra, int n_time) {
        win = w;
        t = w * spectra;
        end = min(t + spectra, n_time);
    }
    __device__ __forceinline__ void next(int spectra, int n_time) {
        t += 16;
        if (t >= end) start(win + 1, spectra, n_time);
    }
};

template <int A, bool kRuns, bool kInt8>
__global__ void __launch_bounds__(kChannelsPerCta * 32)
tracker_stream_kernel(const uint8_t* __restrict__ v, const float* __restrict__ pos,
                      const double* __restrict__ kw, const float* __restrict__ dirs,
                      float* __restrict__ intensity, float* __restrict__ integrated, int n_time,
                      int n_freq, int spectra, int n_windows, int run) {
    constexpr int NW = A / 16;          // 32-bit words per thread per spectrum
    constexpr int kBytes = A / 4;       // bytes per thread per spectrum
    constexpr int kDepth = ring_depth<A>();
    constexpr int kCopy = A == 32 ? 8 : 16, kCopies = kBytes / kCopy;
    constexpr int kSlot = 16 * A;       // bytes of a block: [row half][copy][lane]
    extern __shared__ uint4 smem_raw[];
    uint8_t* ring_all = reinterpret_cast<uint8_t*>(smem_raw);               // [8 warps][kDepth][kSlot] (kRuns)
    uint8_t* parts_all = ring_all + (kRuns ? 8 * kDepth * kSlot : 0);       // [8][part_bytes]
    double* delays = reinterpret_cast<double*>(parts_all + 8 * part_bytes<A, kInt8>());  // [run][A]
    float* stage = reinterpret_cast<float*>(delays + run * A);              // [2][kStageBlocks][16][8], with intensity

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int w_begin = blockIdx.x * run, w_end = min(w_begin + run, n_windows);
    const int f = blockIdx.y * kChannelsPerCta + warp;
    const bool fvalid = f < n_freq;

    // rows g and g + 8 of the block at t, zero past the window's end
    const size_t row_bytes = static_cast<size_t>(n_freq) * A;
    const uint8_t* lane_src = v + static_cast<size_t>(fvalid ? f : 0) * A + q * kBytes;
    auto load_rows = [&](int t, int end, uint32_t (&wd)[2][NW]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool on = fvalid && t + g + 8 * h < end;
            const uint8_t* src = lane_src + static_cast<size_t>(t + g + 8 * h) * row_bytes;
            if constexpr (A == 32) {
                const uint2 x = on ? __ldg(reinterpret_cast<const uint2*>(src)) : make_uint2(0, 0);
                wd[h][0] = x.x; wd[h][1] = x.y;
            } else {
#pragma unroll
                for (int c = 0; c < kCopies; ++c) {
                    const uint4 x = on ? __ldg(reinterpret_cast<const uint4*>(src) + c) : make_uint4(0, 0, 0, 0);
                    wd[h][4 * c] = x.x; wd[h][4 * c + 1] = x.y; wd[h][4 * c + 2] = x.z; wd[h][4 * c + 3] = x.w;
                }
            }
        }
    };
    // the ring: loads of the run's blocks in order, kDepth - 1 ahead
    uint8_t* ring = ring_all + warp * kDepth * kSlot;
    const uint32_t ring_at = static_cast<uint32_t>(__cvta_generic_to_shared(ring)) + lane * kCopy;
    BlockCursor ahead{};
    int ahead_slot = 0;
    auto ring_load = [&]() {
        if (ahead.win < w_end) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = ahead.t + g + 8 * h;
                const bool on = fvalid && t < ahead.end;
                const uint8_t* src = lane_src + (on ? t : ahead.t) * row_bytes;
#pragma unroll
                for (int c = 0; c < kCopies; ++c) {
                    copy_async<kCopy>(ring_at + ahead_slot * kSlot + (h * kCopies + c) * 32 * kCopy, src + c * kCopy, on);
                }
            }
            ahead.next(spectra, n_time);
        }
        if (++ahead_slot == kDepth) ahead_slot = 0;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto ring_read = [&](int slot, uint32_t (&wd)[2][NW]) {
        const uint8_t* src = ring + slot * kSlot + lane * kCopy;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if constexpr (A == 32) {
                const uint2 x = *reinterpret_cast<const uint2*>(src + h * 32 * kCopy);
                wd[h][0] = x.x; wd[h][1] = x.y;
            } else {
#pragma unroll
                for (int c = 0; c < kCopies; ++c) {
                    const uint4 x = *reinterpret_cast<const uint4*>(src + (h * kCopies + c) * 32 * kCopy);
                    wd[h][4 * c] = x.x; wd[h][4 * c + 1] = x.y; wd[h][4 * c + 2] = x.z; wd[h][4 * c + 3] = x.w;
                }
            }
        }
    };

    BlockCursor cur;
    cur.start(w_begin, spectra, n_time);
    uint32_t wa[2][NW], wb[2][NW];
    if constexpr (kRuns) {
        ahead = cur;
#pragma unroll
        for (int i = 0; i < kDepth - 1; ++i) ring_load();
    } else {
        load_rows(cur.t, cur.end, wa);
        load_rows(cur.t + 16, cur.end, wb);
    }
    bool odd = false;
    for (int i = threadIdx.x; i < (w_end - w_begin) * A; i += kChannelsPerCta * 32) {
        const float* d = dirs + 3 * (w_begin + i / A);
        delays[i] = steering_delay(pos, i % A, d[0], d[1], d[2]);
        odd = odd || odd_delay(delays[i]);
    }
    if constexpr (kInt8) odd = __syncthreads_or(odd) != 0; else __syncthreads();

    // B fragments of a window: column g in (re_hi, im_hi, re_lo, im_lo, 0...),
    // or in (re, im) x the four digits.
    const double k = fvalid ? kw[f] : 0.0;
    uint8_t* digits = parts_all + warp * part_bytes<A, kInt8>();
    uint32_t* parts = reinterpret_cast<uint32_t*>(digits);  // rows re_hi, im_hi, re_lo, im_lo of words (a, a + 2)
    uint32_t bfrag[NW][kInt8 ? 1 : 2][2];
    const bool look = kInt8 && (odd || odd_wave_number(k));
    float scale = digit_scale(q);  // of the digit sums; NaN for a window without digits
    auto form_weights = [&](int w) {
        __syncwarp();  // the previous window's words are read
        const double* dl = delays + (w - w_begin) * A;
        if constexpr (kInt8) {
#pragma unroll
            for (int i = 0; i < (A / 2 + 31) / 32; ++i) {
                const int pair = lane + 32 * i;
                if (pair < A / 2) {
                    store_digits<A>(digits, pair, steering_from_delay(k, dl[2 * pair]),
                                    steering_from_delay(k, dl[2 * pair + 1]));
                }
            }
            if (look) scale = weights_have_digits<A>(k, dl, lane) ? digit_scale(q) : NAN;
            __syncwarp();
            uint32_t b[NW][2];
            load_digit_frags<A>(digits, g, q, b);
#pragma unroll
            for (int j = 0; j < NW; ++j) {
                bfrag[j][0][0] = b[j][0];
                bfrag[j][0][1] = b[j][1];
            }
        } else {
#pragma unroll
            for (int i = 0; i < (A / 2 + 31) / 32; ++i) {
                const int word = lane + 32 * i, a0 = 4 * (word >> 1) + (word & 1);
                if (word < A / 2) {
                    const float2 w0 = steering_from_delay(k, dl[a0]), w1 = steering_from_delay(k, dl[a0 + 2]);
#pragma unroll
                    for (int lo = 0; lo < 2; ++lo) {
                        parts[lo * A + word] = split_part(w0.x, lo) | (static_cast<uint32_t>(split_part(w1.x, lo)) << 16);
                        parts[lo * A + A / 2 + word] =
                            split_part(w0.y, lo) | (static_cast<uint32_t>(split_part(w1.y, lo)) << 16);
                    }
                }
            }
            __syncwarp();
            // re: xr * wr - xi * wi; im: xr * wi + xi * wr (column g < 4; the rest are zero)
            const bool is_im = (g & 1) != 0;
            const uint32_t flip = is_im ? 0u : 0x80008000u;
            const uint32_t* row_r = parts + ((g >> 1) & 1) * A + (is_im ? A / 2 : 0) + q * 2 * NW;
            const uint32_t* row_i = parts + ((g >> 1) & 1) * A + (is_im ? 0 : A / 2) + q * 2 * NW;
#pragma unroll
            for (int j = 0; j < NW; j += 2) {
                const uint4 r4 = *reinterpret_cast<const uint4*>(row_r + 2 * j);
                const uint4 i4 = *reinterpret_cast<const uint4*>(row_i + 2 * j);
                const uint32_t wr[4] = {r4.x, r4.y, r4.z, r4.w}, wi[4] = {i4.x, i4.y, i4.z, i4.w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    bfrag[j + (s >> 1)][s & 1][0] = g < 4 ? wr[s] : 0u;
                    bfrag[j + (s >> 1)][s & 1][1] = g < 4 ? wi[s] ^ flip : 0u;
                }
            }
        }
    };

    float acc = 0.f;
    auto stage_powers = [&](int staged, float pow_g, float pow_h) {
        float* st = stage + staged * 16 * kChannelsPerCta + warp;
        st[g * kChannelsPerCta] = pow_g;
        st[(g + 8) * kChannelsPerCta] = pow_h;
    };
    // One block: its spectra's powers into the window sum and the stage.
    auto process = [&](const uint32_t (&wd)[2][NW], int staged) {
        if constexpr (kInt8) {
            int d[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < NW; ++j) {
                mma_16832(d, word_re16(wd[0][j]), word_re16(wd[1][j]), word_im16(wd[0][j]), word_im16(wd[1][j]),
                          bfrag[j][0][0], bfrag[j][0][1]);
            }
            float sq_g, sq_h;
            digit_squares<A>(d, scale, sq_g, sq_h);
            acc = __fadd_rn(acc, __fadd_rn(sq_g, sq_h));  // re^2 and im^2 apart until the window ends
            if (intensity != nullptr) {
                const float pow_g = __fadd_rn(sq_g, __shfl_xor_sync(0xffffffffu, sq_g, 2));
                const float pow_h = __fadd_rn(sq_h, __shfl_xor_sync(0xffffffffu, sq_h, 2));
                if (q == 0) stage_powers(staged, pow_g, pow_h);
            }
        } else {
            float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < NW; ++j) {
                uint32_t re02g, im02g, re13g, im13g, re02h, im02h, re13h, im13h;
                decode_word(wd[0][j], re02g, im02g, re13g, im13g);
                decode_word(wd[1][j], re02h, im02h, re13h, im13h);
                mma_16816(d, re02g, re02h, im02g, im02h, bfrag[j][0][0], bfrag[j][0][1]);
                mma_16816(d, re13g, re13h, im13g, im13h, bfrag[j][1][0], bfrag[j][1][1]);
            }
            // q == 0 holds (re_hi, im_hi), q == 1 holds (re_lo, im_lo) for rows g, g+8.
            float p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = __shfl_xor_sync(0xffffffffu, d[i], 1);
            const float re_g = d[0] + p[0], im_g = d[1] + p[1];
            const float re_h = d[2] + p[2], im_h = d[3] + p[3];
            const float pow_g = re_g * re_g + im_g * im_g;
            const float pow_h = re_h * re_h + im_h * im_h;
            if (q == 0) {
                acc += pow_g + pow_h;
                if (intensity != nullptr) stage_powers(staged, pow_g, pow_h);
            }
        }
    };
    auto finish_window = [&](int w) {
        if (integrated == nullptr) return;
        float sum = acc;
        if constexpr (kInt8) sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        if (lane == 0 && fvalid) integrated[static_cast<size_t>(w) * n_freq + f] = sum;
    };
    // Writes out kStageBlocks staged blocks from `first` on.  One barrier per
    // call: a buffer is written again only after the barrier of the other
    // one, which every thread reaches after its reads here.
    auto write_staged = [&](BlockCursor first, int buf) {
        __syncthreads();
        const int c = threadIdx.x % kChannelsPerCta, fo = blockIdx.y * kChannelsPerCta + c;
        const int r = threadIdx.x / kChannelsPerCta;
        for (int b = 0; b < kStageBlocks && first.win < w_end; ++b) {
            if (r < 16 && first.t + r < first.end && fo < n_freq) {
                intensity[static_cast<size_t>(first.t + r) * n_freq + fo] =
                    stage[((buf * kStageBlocks + b) * 16 + r) * kChannelsPerCta + c];
            }
            first.next(spectra, n_time);
        }
    };

    if constexpr (kRuns) {
        int slot = 0;
        for (int buf = 0; cur.win < w_end; buf ^= 1) {
            const BlockCursor first = cur;
#pragma unroll 1
            for (int b = 0; b < kStageBlocks && cur.win < w_end; ++b) {
                ring_load();
                asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
                if (cur.t == cur.win * spectra) {
                    form_weights(cur.win);
                    acc = 0.f;
                }
                ring_read(slot, wa);
                if (++slot == kDepth) slot = 0;
                process(wa, buf * kStageBlocks + b);
                if (cur.t + 16 >= cur.end) finish_window(cur.win);
                cur.next(spectra, n_time);
            }
            if (intensity != nullptr) write_staged(first, buf);
        }
    } else {
        // the next two blocks' loads are in flight while two blocks compute
        // (blocks are still summed one by one in increasing time)
        form_weights(w_begin);
        BlockCursor first = cur;
        int staged = 0;
        for (; cur.t < cur.end; cur.t += 32) {
            uint32_t na[2][NW], nb[2][NW];
            load_rows(cur.t + 32, cur.end, na);
            load_rows(cur.t + 48, cur.end, nb);
            process(wa, staged);
            if (cur.t + 16 < cur.end) process(wb, staged + 1);  // uniform across the CTA
            if (intensity != nullptr) {
                staged = (staged + 2) % (2 * kStageBlocks);
                if (staged % kStageBlocks == 0 || cur.t + 32 >= cur.end) {
                    write_staged(first, (staged - 1 + 2 * kStageBlocks) % (2 * kStageBlocks) / kStageBlocks);
                    first.t = cur.t + 32;
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int j = 0; j < NW; ++j) {
                    wa[h][j] = na[h][j];
                    wb[h][j] = nb[h][j];
                }
            }
        }
        finish_window(w_begin);
    }
}

template <int A>
bf_status launch_stream(cudaStream_t stream, const uint8_t* v, const float* pos, const double* k, const float* dirs,
                        float* intensity, float* integrated, int T, int F, int S, int W) {
    const int channel_groups = (F + kChannelsPerCta - 1) / kChannelsPerCta;
    const bool runs = S <= kShortWindow;
    // windows per CTA: short windows share a CTA's ramp, as long as the launch
    // fills the GPU; the long form walks one window
    int run = runs ? std::max(1, std::min(kMaxRun, kRunSpectra / S)) : 1;
    while (run > 1 && static_cast<long long>(channel_groups) * ((W + run - 1) / run) < kWantedCtas) run /= 2;
    const bool int8 = S > kHalfWindow;
    const size_t smem = (runs ? 8 * ring_depth<A>() * 16 * A : 0) +
                        8 * (int8 ? part_bytes<A, true>() : part_bytes<A, false>()) + run * A * sizeof(double) +
                        (intensity != nullptr ? 2 * kStageBlocks * 16 * kChannelsPerCta * sizeof(float) : 0);
    auto kernel = !runs  ? tracker_stream_kernel<A, false, true>
                  : int8 ? tracker_stream_kernel<A, true, true>
                         : tracker_stream_kernel<A, true, false>;
    if (smem > 48 * 1024) {  // the limit of a launch that asks for no more; asking costs 0.5 us
        cudaError_t err =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (err != cudaSuccess) return cuda_status(err, "tracker_stream_kernel smem attribute");
    }
    const dim3 grid(static_cast<unsigned>((W + run - 1) / run), static_cast<unsigned>(channel_groups));
    kernel<<<grid, kChannelsPerCta * 32, smem, stream>>>(v, pos, k, dirs, intensity, integrated, T, F, S, W, run);
    return cuda_status(cudaGetLastError(), "tracker_stream_kernel launch");
}

}  // namespace

bf_status launch_tracker_stream(cudaStream_t stream, const uint8_t* v, const float* pos,
                                const double* k, const float* dirs, float* intensity,
                                float* integrated, const bf_dims& d, uint64_t spectra) {
    const uint64_t W = window_count(d.n_time, spectra);
    if (W > 0x7fffffffull || d.n_time > 0x7fffffffull) {
        return set_error(BF_ERR_OVERFLOW, "CUDA tracker grid exceeds the supported size");
    }
    const int T = static_cast<int>(d.n_time), F = static_cast<int>(d.n_freq);
    const int S = static_cast<int>(std::min<uint64_t>(spectra, d.n_time)), w = static_cast<int>(W);
    switch (d.n_ant) {
        case 32: return launch_stream<32>(stream, v, pos, k, dirs, intensity, integrated, T, F, S, w);
        case 64: return launch_stream<64>(stream, v, pos, k, dirs, intensity, integrated, T, F, S, w);
        case 128: return launch_stream<128>(stream, v, pos, k, dirs, intensity, integrated, T, F, S, w);
        case 256: return launch_stream<256>(stream, v, pos, k, dirs, intensity, integrated, T, F, S, w);
        default: return set_error(BF_ERR_INVALID_ARGUMENT, "n_ant must be 32, 64, 128, or 256");
    }
}

}  // namespace bf
