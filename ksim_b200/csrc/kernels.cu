// kernels.cu — sm_100a plain sampling and evaluation kernels.
//
// k_sample: one component per launch, one CTA per tile of blockDim.x shots,
// running sample_tile (sample_tile.cuh): the autoregressive loop of
// kokkos_sim.cpp:214-230 with the term tables staged through shared memory
// by TMA bulk copies.
//
// k_eval: one thread per explicit parameter row, the debug / precision entry
// of kokkos_sim.cpp:157-185 (and the per-term numerator dump).
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/ksim_b200.h"
#include "kernels.h"
#include "sample_tile.cuh"
#include "slice_tile.cuh"
#include "zring.cuh"

namespace ksim {

namespace {

// The kernels without the exact and 64-bit paths fit 96 registers: with
// 128-thread CTAs and 12 KiB staging slots, five CTAs per SM.  The general
// kernel keeps the two-of-256 budget.
#define KSIM_SAMPLE_BOUNDS(P) __maxnreg__((P) != PATHS_ALL ? 96 : 65536 / (256 * KSIM_SAMPLE_MIN_CTAS))
template <int W, bool STAGED, int PATHS = PATHS_ALL>
__global__ void KSIM_SAMPLE_BOUNDS(PATHS) k_sample(const SampleJob j)
{
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bar = (uint64_t *)smem;
    uint8_t *slots = smem + BAR_BYTES;
    if (STAGED) ring_init(bar);
    uint32_t g = 0;
    constexpr int S = shots_per_thread(W);
    uint8_t *scratch = STAGED ? slots + (size_t)NSLOT * j.slot_bytes : slots;
    sample_tile<W, STAGED, false, S, PATHS>(j, (int64_t)blockIdx.x * blockDim.x * S, bar, slots, g,
                                                   scratch);
}

// The sliced sampler: one CTA per `tile` shots (tile <= shots, the width of
// the CTA's bit rows).  S shots a thread; THREADS and CTAS bound the registers.
// EVAL: as slice_tile's.
template <int S, int THREADS, int CTAS, int EVAL>
__global__ void __launch_bounds__(THREADS, CTAS) k_slice(const SampleJob j, const int shots, const int tile)
{
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t *ring = smem + slice_ring_off(j.s_rows, j.s_planes, shots);
    uint64_t *bar = (uint64_t *)ring;
    slice_ring_init(bar);
    uint32_t g = 0;
    const int64_t s0 = (int64_t)blockIdx.x * tile;
    slice_tile<S, false, EVAL>(j, s0, s0 + tile < j.B ? s0 + tile : j.B, shots, smem,
                               slice_rows_bytes(j.s_rows, shots), bar, g);
}

template <int W>
__global__ void __launch_bounds__(128) k_eval(const EvalJob j)
{
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= j.B) return;
    uint64_t v[W];
    const uint8_t *row = j.params + s * j.P;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const int64_t lim = j.P - 64 * w < 64 ? j.P - 64 * w : 64;
        uint64_t x = 0;
        for (int b = 0; b < lim; ++b) x |= (uint64_t)(row[64 * w + b] & 1u) << b;
        v[w] = x;
    }
    set_one_bit<W>(v);
    const GraphDir gd = j.gdir[j.graph];
    const uint8_t *p = j.image + gd.stream_off;
    uint32_t risk = 0;
    if (j.mode == EVAL_TERMS) {
        int64_t *o = (int64_t *)j.out + s * (int64_t)gd.G * 5;
        for (int t = 0; t < gd.G; ++t) {
            const TermHdr h = load_hdr(p);
            TermOut r;
            p = eval_term<W>(p, h, v, r);
            o[5 * t + 0] = (int64_t)r.z.a;
            o[5 * t + 1] = (int64_t)r.z.b;
            o[5 * t + 2] = (int64_t)r.z.c;
            o[5 * t + 3] = (int64_t)r.z.d;
            o[5 * t + 4] = r.pw;
            risk |= r.risk;
        }
    } else {
        double re = 0.0, im = 0.0;
        eval_terms<W>(p, (uint32_t)gd.G, v, re, im, risk);
        double *o = (double *)j.out;
        if (j.mode == EVAL_ABS) {
            o[s] = dsqrt(dadd(dmul(re, re), dmul(im, im)));
        } else {
            o[2 * s] = re;
            o[2 * s + 1] = im;
        }
    }
    if (risk) atomicOr(j.status, (uint32_t)KSIM_FLAG_INT64_RISK);
}

template <int W>
cudaError_t launch_sample_w(const SampleJob &j, const LaunchCfg &cfg, cudaStream_t st)
{
    const int threads = cfg.threads;
    const int64_t tile = (int64_t)threads * shots_per_thread(W);
    const int64_t blocks = (j.B + tile - 1) / tile;
    if (blocks > 0x7FFFFFFF) return cudaErrorInvalidConfiguration;
    const size_t smem = sample_smem_bytes(j.slot_bytes, cfg.staged != 0, W, threads);
    if (cfg.staged && cfg.paths == PATHS_NARROW && W <= 4) {
        cudaError_t e = cudaFuncSetAttribute(k_sample<W, true, PATHS_NARROW>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k_sample<W, true, PATHS_NARROW><<<(unsigned)blocks, threads, smem, st>>>(j);
    } else if (cfg.staged && cfg.paths == PATHS_NARROW_HYBRID && W <= 4) {
        cudaError_t e = cudaFuncSetAttribute(k_sample<W, true, PATHS_NARROW_HYBRID>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        k_sample<W, true, PATHS_NARROW_HYBRID><<<(unsigned)blocks, threads, smem, st>>>(j);
    } else if (cfg.staged) {
        cudaError_t e = cudaFuncSetAttribute(k_sample<W, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
        k_sample<W, true><<<(unsigned)blocks, threads, smem, st>>>(j);
    } else {
        cudaError_t e = cudaFuncSetAttribute(k_sample<W, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
        k_sample<W, false><<<(unsigned)blocks, threads, smem, st>>>(j);
    }
    return cudaGetLastError();
}

template <int S, int THREADS, int CTAS, int EVAL>
cudaError_t launch_slice_as(const SampleJob &j, int shots, int threads, int tile, cudaStream_t st, int *tile_used)
{
    if (tile_used) *tile_used = tile;
    const int64_t blocks = (j.B + tile - 1) / tile;
    if (blocks > 0x7FFFFFFF || !slice_tile_ok(S, shots, threads) || tile > shots) return cudaErrorInvalidConfiguration;
    const int smem = slice_smem_bytes(j.s_rows, j.s_planes, shots);
    cudaError_t e = cudaFuncSetAttribute(k_slice<S, THREADS, CTAS, EVAL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SLICE_SMEM_MAX);
    if (e != cudaSuccess) return e;
    k_slice<S, THREADS, CTAS, EVAL><<<(unsigned)blocks, threads, smem, st>>>(j, shots, tile);
    return cudaGetLastError();
}

// The tile shape by how many SMs the shots can fill.  Measured on the 40-output
// t = 12 program (ms; 512 threads x 1 shot at widths 128 / 256 / 512, 512 x 2
// at 1,024 -- 256 threads x 4, two CTAs an SM -- 256 x 8 at 2,048, two CTAs):
//    10,000 shots  0.195 0.202 0.220                     (18,944 = 148 x 128)
//    37,800        0.387 0.204 0.222 0.275
//    70,000        0.76  0.40  0.226 0.275 0.300
//   100,000        1.14  0.60  0.439 0.275 0.300
//   150,000              0.80  0.446 0.276 0.301 0.506
//   200,000                          0.541 0.405
//   303,104                          0.545 0.405 0.506   (= 296 x 1,024)
//   500,000                                0.793 0.695
// and alike on the 16-output t = 20 one: the widest tile costs least per shot,
// but a narrower one that still fits one wave ends sooner.  Two CTAs of 2,048
// shots need at most 129 parameter rows; with more (60 outputs, F = 100) one
// CTA took 1.318 ms for 606,208 shots, two of 1,024 take 1.002.
// Chunks of at most four terms (eight planes) have work for eight warps in the
// rows pass, and sixteen only wait for one another: with 256 threads 80,000 shots
// of a program of one term a graph and 5, 20, 60 outputs take 24.8, 72.6, 199 us
// (512: 26.2, 75.9, 205), 5,000 shots 16.6, 49.3, 127 (16.8, 50.2, 131); of eight
// terms a graph and 3 outputs 5,000 shots 20.6 (18.6).
template <int EVAL = -1>
cudaError_t launch_slice(const SampleJob &j, const LaunchCfg &cfg, cudaStream_t st, int *tile_used = nullptr)
{
    if (cfg.slice_threads > 0) {  // chosen by the caller: four shots each, a power of two of threads
        const int t = cfg.slice_threads >= 256 ? 256 : cfg.slice_threads >= 128 ? 128 : cfg.slice_threads >= 64 ? 64 : 32;
        return launch_slice_as<4, 256, 2, EVAL>(j, 4 * t, t, 4 * t, st, tile_used);
    }
    const int64_t sms = cfg.sms;
    // (launches of one call overlap: their shape is that of the call's shots, up
    // to the two-per-SM width, which the launches in flight fill together)
    const int64_t n = cfg.call_shots > 0 ? std::min(cfg.call_shots, 2 * sms * 1024) : j.B;
    const bool few = j.s_planes <= 8;
    if (n <= sms * 512) {
        const int shots = n <= sms * 128 ? 128 : n <= sms * 256 ? 256 : 512;
        return launch_slice_as<1, 512, 1, EVAL>(j, shots, few && shots <= 256 ? 256 : 512, shots, st, tile_used);
    }
    if (n <= sms * 1024) {
        if (few) return launch_slice_as<4, 256, 2, EVAL>(j, 1024, 256, 1024, st, tile_used);
        return launch_slice_as<4, 512, 1, EVAL>(j, 1024, 512, 1024, st, tile_used);
    }
    const bool wide = n > 2 * sms * 1024 && slice_two_ctas(j.s_rows, j.s_planes, 2048);
    const int shots = wide ? 2048 : 1024;
    // equal tiles: a last wave that is nearly empty costs as much as a full one
    const int64_t all = cfg.call_shots > 0 ? cfg.call_shots : j.B;
    const int64_t waves = (all + 2 * sms * shots - 1) / (2 * sms * shots);
    const int64_t want = (all + waves * 2 * sms - 1) / (waves * 2 * sms);
    const int tile = (int)((want + 63) / 64 * 64);
    if (wide) return launch_slice_as<8, 256, 2, EVAL>(j, shots, 256, tile, st, tile_used);
    return launch_slice_as<4, 256, 2, EVAL>(j, shots, 256, tile, st, tile_used);
}

template <int W>
cudaError_t launch_eval_w(const EvalJob &j, cudaStream_t st)
{
    const int threads = 128;
    const int64_t blocks = (j.B + threads - 1) / threads;
    if (blocks > 0x7FFFFFFF) return cudaErrorInvalidConfiguration;
    k_eval<W><<<(unsigned)blocks, threads, 0, st>>>(j);
    return cudaGetLastError();
}

// One output byte per thread (grid-stride): HBM-bound byte work.
__global__ void __launch_bounds__(256) k_unpack_bits(const uint8_t *__restrict__ packed, int64_t rows,
                                                     int64_t packed_row, int64_t n_cols, uint8_t *__restrict__ out)
{
    const int64_t n = rows * n_cols;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / n_cols, c = i - r * n_cols;
        out[i] = (packed[r * packed_row + (c >> 3)] >> (c & 7)) & 1u;
    }
}

// One packed byte per thread (grid-stride).
__global__ void __launch_bounds__(256) k_pack_bits(const uint8_t *__restrict__ bytes, int64_t rows, int64_t n_cols,
                                                   int64_t packed_row, uint8_t *__restrict__ out)
{
    const int64_t n = rows * packed_row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / packed_row, b = i - r * packed_row;
        const uint8_t *src = bytes + r * n_cols + 8 * b;
        const int64_t m = n_cols - 8 * b < 8 ? n_cols - 8 * b : 8;
        uint32_t x = 0;
        for (int k = 0; k < m; ++k) x |= (uint32_t)(src[k] & 1u) << k;
        out[i] = (uint8_t)x;
    }
}

unsigned byte_grid(int64_t n)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t want = (n + 255) / 256;
    const int64_t cap = (int64_t)sms * 8;
    return (unsigned)(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace

cudaError_t launch_unpack_bits(const uint8_t *packed, int64_t rows, int64_t packed_row, int64_t n_cols, uint8_t *out,
                               cudaStream_t st)
{
    if (rows <= 0 || n_cols <= 0) return cudaSuccess;
    k_unpack_bits<<<byte_grid(rows * n_cols), 256, 0, st>>>(packed, rows, packed_row, n_cols, out);
    return cudaGetLastError();
}

cudaError_t launch_pack_bits(const uint8_t *bytes, int64_t rows, int64_t n_cols, int64_t packed_row, uint8_t *out,
                             cudaStream_t st)
{
    if (rows <= 0 || n_cols <= 0) return cudaSuccess;
    k_pack_bits<<<byte_grid(rows * packed_row), 256, 0, st>>>(bytes, rows, n_cols, packed_row, out);
    return cudaGetLastError();
}

size_t staged_smem_bytes(int slot_bytes) { return (size_t)BAR_BYTES + (size_t)NSLOT * (size_t)slot_bytes; }

cudaError_t launch_sample(const SampleJob &job, int W, const LaunchCfg &cfg, cudaStream_t st)
{
    if (job.B <= 0) return cudaSuccess;
    if (cfg.threads <= 0 || cfg.threads > 256 || (cfg.threads & 31)) return cudaErrorInvalidConfiguration;
    if (cfg.sliced) return launch_slice(job, cfg, st);
    switch (W) {
    case 1: return launch_sample_w<1>(job, cfg, st);
    case 2: return launch_sample_w<2>(job, cfg, st);
    case 3: return launch_sample_w<3>(job, cfg, st);
    case 4: return launch_sample_w<4>(job, cfg, st);
    case 5: return launch_sample_w<5>(job, cfg, st);
    case 6: return launch_sample_w<6>(job, cfg, st);
    case 8: return launch_sample_w<8>(job, cfg, st);
    case 10: return launch_sample_w<10>(job, cfg, st);
    case 12: return launch_sample_w<12>(job, cfg, st);
    case 16: return launch_sample_w<16>(job, cfg, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_eval_sliced(const SampleJob &job, int mode, const LaunchCfg &cfg, cudaStream_t st, int *tile)
{
    if (job.B <= 0) return cudaSuccess;
    return mode == EVAL_ABS ? launch_slice<EVAL_ABS>(job, cfg, st, tile)
                            : launch_slice<EVAL_COMPLEX>(job, cfg, st, tile);
}

cudaError_t launch_eval(const EvalJob &job, int W, cudaStream_t st)
{
    if (job.B <= 0) return cudaSuccess;
    switch (W) {
    case 1: return launch_eval_w<1>(job, st);
    case 2: return launch_eval_w<2>(job, st);
    case 3: return launch_eval_w<3>(job, st);
    case 4: return launch_eval_w<4>(job, st);
    case 5: return launch_eval_w<5>(job, st);
    case 6: return launch_eval_w<6>(job, st);
    case 8: return launch_eval_w<8>(job, st);
    case 10: return launch_eval_w<10>(job, st);
    case 12: return launch_eval_w<12>(job, st);
    case 16: return launch_eval_w<16>(job, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace ksim
