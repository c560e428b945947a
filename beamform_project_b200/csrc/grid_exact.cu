// grid_exact.cu -- fixed-grid beamformer in the reference's float32 order.
//
// This is the plain drop-in for launch_packed_beamformer and
// launch_packed_integrated_beamformer (reference include/beamformer/
// cuda_stage_api.hpp:21-35, kernels src/cuda_beamformer.cu:108-354).  Each
// output is the same sequence of correctly rounded float32 operations as
// cpu_beamform_packed_intensity (src/cpu_beamformer.cpp:56-78) followed by
// cpu_integrate_intensity (src/temporal_integration.cpp:95-109), so results
// are bit-identical to the reference CPU core built without FMA contraction.
//
// Work decomposition (not the reference's): a CTA of 8 warps owns one
// (channel, group of up to 64 beams, run of whole windows) and walks the run
// in tiles of 64 spectra.  A warp owns 8 spectra of the tile and every beam
// of the group: lane = (one of 8 beam columns, one of 4 spectrum pairs), with
// BL beams per lane.  (Short blocks take CTAs of 2 warps and tiles of 16
// spectra, where a warp without spectra does no arithmetic: one spectrum of
// 128 beams at 64 antennas 26.6 us, 65.5 with the tile of 64.)  Two beams at a
// time share packed f32x2 registers, so a complex multiply-add of two beams is
// eight packed instructions, each rounding its halves as the scalar
// instruction would; the last beam of an odd BL packs the pair's two spectra
// instead.  Weights sit in shared memory
// as (re, re, im, im) of two beams and voltages as (re, re, im, im) of two
// spectra per antenna: BL / 2 + 1 loads of 16 bytes per lane feed 8 BL packed
// instructions.  The weights stay for the CTA's life (32 beams a group at 256
// antennas, so that two CTAs fit an SM); voltages are staged 64 antennas at a
// time, the sums staying in registers.
//
// What bounds it: the order of roundings forbids fused multiply-adds, so a
// complex multiply-add is eight operations on a pipe that does 128 per SM and
// clock (scalar or packed alike, measured 124-127); packing halves the
// instructions, which leaves issue slots to the loads.  A 16-byte load takes
// the shared-memory port for four clocks whatever its lanes share, so what
// each brings counts: with one beam per load, weights doubled in shared
// memory, the port was full (6.0 ms for the shape below).
// Measured, 64 antennas, 15360 spectra, 64 beams, windows of 320: 5.60 ms,
// 81 % of the pipe's rate (8.45 ms with scalar arithmetic, a warp's lanes one
// beam each and four spectra at a time); 37 beams per spectrum, 1000 spectra:
// 0.273 ms (0.597 ms, most of it for the second 32-beam tile's idle lanes).
// The powers of a tile go through shared memory: a thread per beam then adds
// them to its window sum strictly in increasing time, or the CTA writes them
// out row by row.
#include "bf_internal.cuh"
#include "packed_f32.cuh"

namespace bf {
namespace {

constexpr int kWarps = 8;             // warps of a CTA, and of one for a short block
constexpr int kShortWarps = 2;
constexpr int tile_spectra(int warps) { return 8 * warps; }  // four pairs per warp
constexpr int kTile = tile_spectra(kWarps);
constexpr int kChunk = 64;            // antennas staged at once
// Longest block of the short form: its CTAs are a quarter of the size, so more
// of them hide one another's latency while most of a 64-spectrum tile would be
// empty.  64 beams, 64 antennas: 16 spectra 16.4 us (30.7 in the long form), 32
// 24.6 (32.2); 128 antennas 16 28.7 (49.2), but 32 of 128 beams 93.9 (86.1: two
// tiles per CTA, and the weights leave room for five on an SM).
__host__ __device__ constexpr int short_block(uint64_t n_ant) { return n_ant <= 64 ? 32 : 16; }
// Beams per CTA: up to 64, with the weights of every antenna in half an SM's
// shared memory.
__host__ __device__ constexpr int max_group(uint64_t n_ant) { return n_ant <= 128 ? 64 : 32; }
// Spectra per CTA: enough tiles to cover the staging of the weights; fewer,
// then fewer beams, while the launch has under four rounds of CTAs (two per SM).
constexpr int kUnitSpectra = 5 * kTile, kWantedCtas = 4 * 2 * 148;

struct ExactParams {
    const uint8_t* v;
    const float2* w;
    float* out;
    int n_time, n_freq, n_ant, n_beams;
    int tiled, spectra;     // spectra per window; 0: per-spectrum output
    int unit_len, groups;   // spectra per CTA (whole windows), beam groups of 8 BL
    float one;              // 1
};

template <int BL, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) grid_exact_kernel(const ExactParams p) {
    constexpr int kThreads = 32 * WARPS, kTile = tile_spectra(WARPS), kPairs = kTile / 2;
    constexpr int kBeams = 8 * BL;
    constexpr int JP = BL / 2;             // beam pairs per lane: beams 16 j + 2 col and the next
    constexpr bool kOdd = (BL & 1) != 0;   // and beam 16 JP + col
    constexpr int kPwPitch = kBeams + 4;   // the four pairs of a store land in different banks
    const int AC = min(p.n_ant, kChunk);
    extern __shared__ float4 smem[];
    // [A][kBeams] float2: (re, re, im, im) of two beams, pair j of antenna a
    // at j ^ (a % 8) so that stores along the antennas spread over the banks
    float2* ws = reinterpret_cast<float2*>(smem);
    float4* xs = smem + p.n_ant * kBeams / 2;                    // [kPairs][AC], antenna a at a ^ (pair % 4)
    float* pw = reinterpret_cast<float*>(xs + kPairs * AC);  // [kTile][kPwPitch]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = lane & 7, pair = 4 * warp + (lane >> 3);
    const int f = blockIdx.x % p.n_freq;
    const int rest = blockIdx.x / p.n_freq;
    const int b0 = (rest % p.groups) * kBeams;
    const int unit = rest / p.groups;
    const int t_begin = unit * p.unit_len;
    const int t_end = min(t_begin + p.unit_len, p.n_time);
    const int chunks = p.n_ant / AC;
    const int steps = (t_end - t_begin + kTile - 1) / kTile * chunks;

    {
        constexpr int kBatch = 8;  // loads in flight per thread
        const int n = p.n_ant * kBeams, beam_tiles = (p.n_beams + 31) / 32;
        for (int i0 = threadIdx.x; i0 < n; i0 += kBatch * kThreads) {
            float2 x[kBatch];
            // lanes run along the antennas (canonical weights) or the beams (tiled): coalesced loads
            auto at = [&](int k, int& a, int& lb) {
                const int i = i0 + k * kThreads;
                a = p.tiled ? i / kBeams : i % p.n_ant;
                lb = p.tiled ? i % kBeams : i / p.n_ant;
                return i < n;
            };
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                int a, lb;
                x[k] = make_float2(0.f, 0.f);
                if (!at(k, a, lb) || b0 + lb >= p.n_beams) continue;
                const int b = b0 + lb;
                x[k] = p.tiled ? p.w[((static_cast<size_t>(f) * beam_tiles + b / 32) * p.n_ant + a) * 32 + b % 32]
                               : p.w[(static_cast<size_t>(b) * p.n_freq + f) * p.n_ant + a];
            }
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                int a, lb;
                if (!at(k, a, lb)) continue;
                float2* row = ws + a * kBeams;
                if (lb < 16 * JP) {
                    float* two = reinterpret_cast<float*>(row + 2 * ((lb >> 1) ^ (a & 7)));
                    two[lb & 1] = x[k].x;
                    two[2 + (lb & 1)] = x[k].y;
                } else {
                    row[lb] = x[k];
                }
            }
        }
    }
    // A thread's words of a step: 4 antennas of the two spectra of a pair,
    // one or two such items (256 or 512 per step).
    const int words = AC / 4;
    uint32_t pre[2][2];
    auto load_voltage = [&](int step) {
        const int tb = t_begin + step / chunks * kTile, a0 = step % chunks * AC;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = threadIdx.x + k * kThreads;
            const int t = tb + 2 * (i / words);
            const uint8_t* src = p.v + (static_cast<size_t>(t) * p.n_freq + f) * p.n_ant + a0 + 4 * (i % words);
            const size_t row = static_cast<size_t>(p.n_freq) * p.n_ant;
            const bool on = i < kPairs * words && step < steps;
            pre[k][0] = on && t < t_end ? __ldg(reinterpret_cast<const uint32_t*>(src)) : 0u;
            pre[k][1] = on && t + 1 < t_end ? __ldg(reinterpret_cast<const uint32_t*>(src + row)) : 0u;
        }
    };
    auto store_voltage = [&]() {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = threadIdx.x + k * kThreads;
            if (i >= kPairs * words) break;
            const int pr = i / words, wd = i % words;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int a = (j + (wd >> 1)) & 3;  // rotated: eight lanes store to different banks
                xs[pr * AC + 4 * wd + (a ^ (pr & 3))] =
                    make_float4(nibble_float(pre[k][0], 8 * a), nibble_float(pre[k][1], 8 * a),
                                nibble_float(pre[k][0], 8 * a + 4), nibble_float(pre[k][1], 8 * a + 4));
            }
        }
    };
    // Takes the finished tile's powers: window sums (thread = beam) or rows.
    const int lb = threadIdx.x;
    float acc = 0.f;
    int left = p.spectra, win = p.spectra > 0 ? t_begin / p.spectra : 0;
    auto finish_window = [&]() {
        if (b0 + lb < p.n_beams) p.out[(static_cast<size_t>(win) * p.n_freq + f) * p.n_beams + b0 + lb] = acc;
        acc = 0.f;
        left = p.spectra;
        ++win;
    };
    auto take_powers = [&](int tb) {
        const int n = min(kTile, t_end - tb);
        if (p.spectra > 0) {
            if (lb >= kBeams) return;
            const float* src = pw + lb;
            for (int t = 0; t < n;) {
                const int len = min(n - t, left);
#pragma unroll 8
                for (int i = 0; i < len; ++i) acc = __fadd_rn(acc, src[(t + i) * kPwPitch]);
                t += len;
                left -= len;
                if (left == 0) finish_window();
            }
        } else {
            const int nb = min(kBeams, p.n_beams - b0);
            for (int i = threadIdx.x; i < n * kBeams; i += kThreads) {
                const int t = i / kBeams, b = i % kBeams;
                if (b < nb) {
                    p.out[(static_cast<size_t>(tb + t) * p.n_freq + f) * p.n_beams + b0 + b] = pw[t * kPwPitch + b];
                }
            }
        }
    };

    load_voltage(0);
    uint64_t sr[2][JP + 1], si[2][JP + 1];  // [spectrum of the pair][beam pair]; [0][JP]: the odd beam
    const uint64_t plus = pack2(p.one, p.one), minus = pack2(-p.one, -p.one);
    auto cmac = [&](uint64_t& re, uint64_t& im, uint64_t wr, uint64_t wi, uint64_t xr, uint64_t xi) {
        re = add2(re, fma2(mul2(wi, xi), minus, mul2(wr, xr)));
        im = add2(im, fma2(mul2(wi, xr), plus, mul2(wr, xi)));
    };
    for (int step = 0; step < steps; ++step) {
        const int chunk = step % chunks;
        __syncthreads();  // the previous step's operands are read, its tile's powers written
        store_voltage();
        load_voltage(step + 1);
        if (step > 0 && chunk == 0) take_powers(t_begin + (step / chunks - 1) * kTile);
        __syncthreads();
        if (chunk == 0) {
#pragma unroll
            for (int j = 0; j <= JP; ++j) sr[0][j] = sr[1][j] = si[0][j] = si[1][j] = 0;
        }
        // the warp's four pairs read antenna a from four different bank groups
        const float4* xrow = xs + pair * AC;
        // a warp without spectra in the tile (in the long form the test costs more
        // than it saves: 1 % of long blocks)
        if (WARPS == kShortWarps && t_begin + step / chunks * kTile + 8 * warp >= t_end) continue;
#pragma unroll 1
        for (int a0 = 0; a0 < AC; a0 += 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x4 = xrow[a0 + (i ^ (pair & 3))];
                const float2* wrow = ws + (chunk * AC + a0 + i) * kBeams;
                const uint64_t xr[2] = {pack2(x4.x, x4.x), pack2(x4.y, x4.y)};
                const uint64_t xi[2] = {pack2(x4.z, x4.z), pack2(x4.w, x4.w)};
#pragma unroll
                for (int j = 0; j < JP; ++j) {
                    const float4 w4 = reinterpret_cast<const float4*>(wrow)[8 * j + (col ^ i)];
                    const uint64_t wr = pack2(w4.x, w4.y), wi = pack2(w4.z, w4.w);
#pragma unroll
                    for (int u = 0; u < 2; ++u) cmac(sr[u][j], si[u][j], wr, wi, xr[u], xi[u]);
                }
                if constexpr (kOdd) {
                    const float2 w = wrow[16 * JP + col];
                    cmac(sr[0][JP], si[0][JP], pack2(w.x, w.x), pack2(w.y, w.y), pack2(x4.x, x4.y),
                         pack2(x4.z, x4.w));
                }
            }
        }
        if (chunk + 1 == chunks) {
            auto power = [&](int u, int j) {
                return unpack2(fma2(mul2(si[u][j], si[u][j]), plus, mul2(sr[u][j], sr[u][j])));
            };
            float* dst = pw + 2 * pair * kPwPitch;
#pragma unroll
            for (int j = 0; j < JP; ++j) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const F2 two = power(u, j);
                    *reinterpret_cast<float2*>(dst + u * kPwPitch + 16 * j + 2 * col) = make_float2(two.x, two.y);
                }
            }
            if constexpr (kOdd) {
                const F2 two = power(0, JP);
                dst[16 * JP + col] = two.x;
                dst[kPwPitch + 16 * JP + col] = two.y;
            }
        }
    }
    __syncthreads();
    take_powers(t_begin + (steps / chunks - 1) * kTile);
    if (p.spectra > 0 && lb < kBeams && left < p.spectra) finish_window();  // partial last window
}

template <int BL, int WARPS>
bf_status launch_exact(cudaStream_t stream, const ExactParams& p, unsigned blocks) {
    const int AC = p.n_ant < kChunk ? p.n_ant : kChunk;
    const int smem = (p.n_ant * 4 * BL + tile_spectra(WARPS) / 2 * AC) * static_cast<int>(sizeof(float4)) +
                     tile_spectra(WARPS) * (8 * BL + 4) * static_cast<int>(sizeof(float));
    cudaError_t err =
        cudaFuncSetAttribute(grid_exact_kernel<BL, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return cuda_status(err, "grid_exact_kernel smem attribute");
    grid_exact_kernel<BL, WARPS><<<blocks, 32 * WARPS, smem, stream>>>(p);
    return cuda_status(cudaGetLastError(), "grid_exact_kernel launch");
}

template <int BL>
bf_status launch_beams(int bl, cudaStream_t stream, const ExactParams& p, unsigned blocks) {
    if constexpr (BL > 8) {
        return set_error(BF_ERR_LOGIC, "beam group out of range");
    } else {
        if (bl != BL) return launch_beams<BL + 1>(bl, stream, p, blocks);
        return p.n_time <= short_block(p.n_ant) ? launch_exact<BL, kShortWarps>(stream, p, blocks)
                                                : launch_exact<BL, kWarps>(stream, p, blocks);
    }
}

}  // namespace

bf_status launch_grid_exact(int kernel, cudaStream_t stream, const uint8_t* v, const float* w,
                            float* out, const bf_dims& d, uint64_t spectra, bool integrate) {
    const uint64_t S = integrate ? spectra : 1;
    if (window_count(d.n_time, integrate ? spectra : 32) > (1ull << 31) / 4 || d.n_time > (1ull << 31) - 1024) {
        return set_error(BF_ERR_OVERFLOW, "CUDA grid exceeds the supported size");
    }
    uint64_t groups = (d.n_beams + max_group(d.n_ant) - 1) / max_group(d.n_ant);
    uint64_t unit = kUnitSpectra;
    while (unit > kTile && groups * d.n_freq * window_count(d.n_time, unit) < kWantedCtas) unit -= kTile;
    unit = S * (unit / S > 0 ? unit / S : 1);
    if (unit > d.n_time) unit = d.n_time;
    while (16 * groups < d.n_beams && groups * d.n_freq * window_count(d.n_time, unit) < kWantedCtas) ++groups;
    const uint64_t bl = ((d.n_beams + groups - 1) / groups + 7) / 8;
    groups = (d.n_beams + 8 * bl - 1) / (8 * bl);
    const uint64_t blocks = groups * d.n_freq * window_count(d.n_time, unit);
    if (blocks > 0x7fffffffull) return set_error(BF_ERR_OVERFLOW, "CUDA grid exceeds the supported size");
    ExactParams p{};
    p.v = v;
    p.w = reinterpret_cast<const float2*>(w);
    p.out = out;
    p.n_time = static_cast<int>(d.n_time);
    p.n_freq = static_cast<int>(d.n_freq);
    p.n_ant = static_cast<int>(d.n_ant);
    p.n_beams = static_cast<int>(d.n_beams);
    p.tiled = kernel == BF_KERNEL_TILED;
    p.spectra = integrate ? static_cast<int>(spectra < d.n_time ? spectra : d.n_time) : 0;
    p.unit_len = static_cast<int>(unit);
    p.groups = static_cast<int>(groups);
    p.one = 1.0f;
    return launch_beams<1>(static_cast<int>(bl), stream, p, static_cast<unsigned>(blocks));
}

}  // namespace bf
