// Small helper kernels: dequantisation dump (parity check of the unpack rule),
// arg-max over fp16 logits, L2 flush for cold timing.
#include <cuda_fp16.h>
#include <float.h>

#include <atomic>

#include "kernels.h"
#include "ptx.cuh"

namespace nnb {
namespace {

__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }

// out[n,k] = float(code) * float(scale): the unpack contract of
// src/models/lfm2-5-350m/kernels/gemv_m1_q4.cl:31-40 (nibble - 8, low nibble = even k)
// and src/models/lfm2-5-350m/scripts/quantize_weights.py:136 (int8 * per-row scale).
template <int FMT>
__global__ void dequant_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ scale, float* __restrict__ out,
                               int N, int K) {
    const size_t total = (size_t)N * K;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t n = i / K;
        const int k = (int)(i - n * K);
        float v;
        if (FMT == FMT_FP16) {
            v = h2f(reinterpret_cast<const uint16_t*>(W)[i]);
        } else if (FMT == FMT_INT8) {
            v = (float)reinterpret_cast<const int8_t*>(W)[i] * h2f(scale[n]);
        } else {
            const uint8_t b = W[n * (size_t)(K / 2) + (k >> 1)];
            const int code = (int)((b >> (4 * (k & 1))) & 0xF) - 8;
            v = (float)code * h2f(scale[n * (size_t)(K / 32) + (k >> 5)]);
        }
        out[i] = v;
    }
}

// Order-preserving key: larger value wins, then the LOWER index.
__device__ __forceinline__ unsigned long long argmax_key(float v, int idx) {
    unsigned int b = __float_as_uint(v);
    b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return ((unsigned long long)b << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned int)idx);
}

// One launch: every block folds its values into `slot` (0 between launches) and the block that finishes last writes the index and
// clears the words.  (Clearing, folding and finishing as three launches cost a step of one token 6 us on a 151936-entry
// vocabulary, most of it launches.)
__global__ void __launch_bounds__(256) argmax_half_kernel(const uint16_t* __restrict__ v, int n, unsigned long long* slot, unsigned* done, int* out_idx) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    unsigned long long best = 0ull;
    auto take = [&](uint16_t h, int i) {
        const float f = h2f(h);
        if (f == f) {  // NaNs never win
            const unsigned long long k = argmax_key(f, i);
            best = k > best ? k : best;
        }
    };
    const int stride = gridDim.x * blockDim.x, at = blockIdx.x * blockDim.x + threadIdx.x;
    const int pieces = (reinterpret_cast<uintptr_t>(v) & 15) == 0 ? n / 8 : 0;
    for (int p = at; p < pieces; p += stride) {
        const uint4 q = reinterpret_cast<const uint4*>(v)[p];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            take((uint16_t)(w[j] & 0xFFFFu), p * 8 + 2 * j);
            take((uint16_t)(w[j] >> 16), p * 8 + 2 * j + 1);
        }
    }
    for (int i = pieces * 8 + at; i < n; i += stride) take(v[i], i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
    }
    __shared__ unsigned long long sm[8];
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < 8; ++i) best = sm[i] > best ? sm[i] : best;
        if (best) atomicMax(slot, best);
        __threadfence();
        if (atomicAdd(done, 1u) == gridDim.x - 1u) {
            __threadfence();
            const unsigned long long k = *reinterpret_cast<volatile unsigned long long*>(slot);
            *reinterpret_cast<volatile unsigned long long*>(slot) = 0ull;
            *reinterpret_cast<volatile unsigned*>(done) = 0u;
            *out_idx = k ? (int)(0xFFFFFFFFu - (unsigned int)(k & 0xFFFFFFFFull)) : -1;
        }
    }
}

// RMSNorm on fp16 storage, one block per row: out = half((x * rsqrt(mean(x^2) + eps)) * weight)
// (src/models/smollm2-135m-instruct/kernels/rmsnorm.cl:27-104; fp32 sums, a different but fixed order).
__global__ void rmsnorm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, uint16_t* __restrict__ out, int cols, float eps) {
    const uint16_t* xr = x + (size_t)blockIdx.x * cols;
    uint16_t* orow = out + (size_t)blockIdx.x * cols;
    float ss = 0.f;
    for (int c = threadIdx.x; c < cols; c += blockDim.x) {
        const float v = h2f(xr[c]);
        ss += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    __shared__ float part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += part[i];
    const float inv = 1.0f / sqrtf(tot / (float)cols + eps);
    for (int c = threadIdx.x; c < cols; c += blockDim.x) orow[c] = __half_as_ushort(__float2half_rn((h2f(xr[c]) * inv) * h2f(w[c])));
}

// The same for rows of whole, aligned 16-byte pieces: a warp per row, the row kept in registers between the sum and the scaling
// (up to NORM_PIECES * 256 values; beyond that it is read again), launched so that the projection that follows sets up and
// fetches weights meanwhile.  It moves 4 bytes per value and is bound by its own latency: 512 x 896 took 5.6 us as one block
// per row with two-byte accesses and a plain launch.
constexpr int NORM_WARPS = 4, NORM_PIECES = 8;
__global__ void __launch_bounds__(NORM_WARPS * 32) rmsnorm_rows_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w,
                                                                      uint16_t* __restrict__ out, int rows, int cols, float eps) {
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, r = blockIdx.x * NORM_WARPS + (threadIdx.x >> 5), pieces = cols / 8;
    const uint4* gw = reinterpret_cast<const uint4*>(w);
    pdl_wait_prior_grid();   // the rows, and as far as is known the norm weight, may come from the launch before
    if (r >= rows) return;
    const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)r * cols);
    const uint4 g0 = lane < pieces ? gw[lane] : make_uint4(0, 0, 0, 0);   // (asked for with the row)
    uint4* orow = reinterpret_cast<uint4*>(out + (size_t)r * cols);
    uint4 v[NORM_PIECES];
#pragma unroll
    for (int j = 0; j < NORM_PIECES; ++j) v[j] = lane + j * 32 < pieces ? xr[lane + j * 32] : make_uint4(0, 0, 0, 0);
    float ss = 0.f;
    auto add = [&](const uint4& q) {
        const uint32_t q4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&q4[i]));
            ss += f.x * f.x;
            ss += f.y * f.y;
        }
    };
#pragma unroll
    for (int j = 0; j < NORM_PIECES; ++j) add(v[j]);
    for (int p = lane + NORM_PIECES * 32; p < pieces; p += 32) add(xr[p]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.0f / sqrtf(ss / (float)cols + eps);
    auto scaled = [&](const uint4& q, const uint4& g) {
        const uint32_t q4[4] = {q.x, q.y, q.z, q.w}, g4[4] = {g.x, g.y, g.z, g.w};
        uint32_t o4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 fx = __half22float2(*reinterpret_cast<const __half2*>(&q4[i])), fg = __half22float2(*reinterpret_cast<const __half2*>(&g4[i]));
            const __half2 h = __floats2half2_rn((fx.x * inv) * fg.x, (fx.y * inv) * fg.y);
            o4[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        return make_uint4(o4[0], o4[1], o4[2], o4[3]);
    };
#pragma unroll
    for (int j = 0; j < NORM_PIECES; ++j)
        if (lane + j * 32 < pieces) orow[lane + j * 32] = scaled(v[j], j == 0 ? g0 : gw[lane + j * 32]);
    for (int p = lane + NORM_PIECES * 32; p < pieces; p += 32) orow[p] = scaled(xr[p], gw[p]);
}

// out[r][c] = half(float(out[r][c]) + float(bias[c])) for up to three (out, bias) pairs of one launch:
// bias_add_rowmajor, src/models/qwen2-5-0-5b/kernels/bias_add.cl:18-40 (the projection's result is
// rounded to fp16 first, then the bias is added in fp32 and the sum rounded again, as there).
__global__ void bias_add_kernel(BiasArgs a) {
    const int seg = blockIdx.y;
    uint16_t* out = a.out[seg];
    const uint16_t* bias = a.bias[seg];
    const int cols = a.cols[seg];
    const long long total = (long long)a.rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i % cols);
        out[i] = __half_as_ushort(__float2half_rn(h2f(out[i]) + h2f(bias[c])));
    }
}

// Read-bandwidth probes: what the weight streams of this library can reach at best on this GPU
// (the role of gemv_stream_buf / gemv_stream_img, src/models/lfm2-5-350m/kernels/gemv_m1.cl:537-589,
// driven by run_bw_probe, src/models/lfm2-5-350m/src/main.cpp:29-139).  The two read paths of this
// hardware stand where the reference has buffer and image reads: 16-byte loads by every thread, and
// bulk copies into shared memory by the TMA unit (the path the streaming kernels use).
__global__ void __launch_bounds__(256) probe_loads_kernel(const uint4* __restrict__ src, size_t n16, float* __restrict__ sink) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    unsigned int acc = 0u;
    constexpr int U = 8;  // independent loads in flight per thread
    for (; i + (U - 1) * stride < n16; i += U * stride) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v[u].x), "=r"(v[u].y), "=r"(v[u].z), "=r"(v[u].w)
                         : "l"(src + i + u * stride));
#pragma unroll
        for (int u = 0; u < U; ++u) acc += v[u].x ^ v[u].y ^ v[u].z ^ v[u].w;
    }
    for (; i < n16; i += stride) {
        const uint4 v = src[i];
        acc += v.x ^ v.y ^ v.z ^ v.w;
    }
    if (acc == 0x9E3779B9u) sink[threadIdx.x] = 1.f;  // keeps the loads alive; practically never taken
}

constexpr int PROBE_CHUNK = 16384;
constexpr int PROBE_STAGES = 8;

__global__ void __launch_bounds__(32) probe_tma_kernel(const uint8_t* __restrict__ src, size_t nchunks, unsigned* __restrict__ status) {
    extern __shared__ __align__(128) uint8_t probe_smem[];
    __shared__ __align__(8) uint64_t bars[PROBE_STAGES];
    if (threadIdx.x != 0) return;
    for (int s = 0; s < PROBE_STAGES; ++s) mbar_init(smem_u32(&bars[s]), 1);
    mbar_init_fence();
    const uint64_t pol = l2_policy_evict_first();
    size_t issued = 0, waited = 0;   // per stage ring: copy number i lands in stage i % PROBE_STAGES
    bool ok = true;
    for (size_t c = blockIdx.x; c < nchunks && ok; c += gridDim.x) {
        if (issued >= PROBE_STAGES) {  // the copy that used this stage before must have landed
            ok = mbar_wait_bounded(smem_u32(&bars[waited % PROBE_STAGES]), (uint32_t)((waited / PROBE_STAGES) & 1));
            if (!ok) break;
            ++waited;
        }
        const int s = (int)(issued % PROBE_STAGES);
        mbar_arrive_expect_tx(smem_u32(&bars[s]), PROBE_CHUNK);
        bulk_g2s(smem_u32(probe_smem + (size_t)s * PROBE_CHUNK), src + c * (size_t)PROBE_CHUNK, PROBE_CHUNK, smem_u32(&bars[s]), pol);
        ++issued;
    }
    // every copy in flight lands before the block gives its shared memory back (bounded as well)
    for (; waited < issued; ++waited)
        if (!mbar_wait_bounded(smem_u32(&bars[waited % PROBE_STAGES]), (uint32_t)((waited / PROBE_STAGES) & 1))) ok = false;
    if (!ok) atomicExch(status, 1u);
}

__global__ void l2_flush_kernel(uint4* buf, size_t n16) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x) {
        uint4 v = buf[i];
        v.x += 1u;
        buf[i] = v;
    }
}

}  // namespace

int current_sm_count() {
    static std::atomic<int> cached[64] = {};   // (any thread; all find the same number)
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 132;
    int n = cached[dev].load(std::memory_order_relaxed);
    if (!n) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 132;
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

cudaError_t launch_dequant(int fmt, int N, int K, const void* W, const uint16_t* scale, float* out, cudaStream_t st) {
    const size_t total = (size_t)N * K;
    if (total == 0) return cudaSuccess;
    const int threads = 256;
    size_t blocks = (total + threads - 1) / threads;
    const size_t cap = (size_t)current_sm_count() * 16;
    if (blocks > cap) blocks = cap;
    const uint8_t* w = static_cast<const uint8_t*>(W);
    if (fmt == FMT_FP16) dequant_kernel<FMT_FP16><<<(unsigned)blocks, threads, 0, st>>>(w, scale, out, N, K);
    else if (fmt == FMT_INT8) dequant_kernel<FMT_INT8><<<(unsigned)blocks, threads, 0, st>>>(w, scale, out, N, K);
    else dequant_kernel<FMT_Q4><<<(unsigned)blocks, threads, 0, st>>>(w, scale, out, N, K);
    return cudaGetLastError();
}

cudaError_t launch_argmax_half(const uint16_t* v, int n, int* out_idx, unsigned long long* slot, unsigned* done, cudaStream_t st, bool pdl) {
    int blocks = (n + 2047) / 2048;   // one 16-byte piece per thread, up to one block per SM
    const int cap = current_sm_count();
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, argmax_half_kernel, v, n, slot, done, out_idx);
}

cudaError_t launch_rmsnorm(const uint16_t* x, const uint16_t* w, uint16_t* out, int rows, int cols, float eps, cudaStream_t st, bool pdl) {
    if (rows <= 0 || cols <= 0) return cudaSuccess;
    if (cols % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((rows + NORM_WARPS - 1) / NORM_WARPS));
        cfg.blockDim = dim3(NORM_WARPS * 32);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, rmsnorm_rows_kernel, x, w, out, rows, cols, eps);
    }
    rmsnorm_kernel<<<(unsigned)rows, 256, 0, st>>>(x, w, out, cols, eps);
    return cudaGetLastError();
}

cudaError_t launch_bias_add(const BiasArgs& a, cudaStream_t st) {
    if (a.rows <= 0 || a.nseg <= 0) return cudaSuccess;
    int maxc = 0;
    for (int i = 0; i < a.nseg; ++i) maxc = a.cols[i] > maxc ? a.cols[i] : maxc;
    long long blocks = ((long long)a.rows * maxc + 255) / 256;
    const long long cap = (long long)current_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    bias_add_kernel<<<dim3((unsigned)blocks, (unsigned)a.nseg), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_probe_loads(const void* src, size_t bytes, float* sink, cudaStream_t st) {
    probe_loads_kernel<<<current_sm_count() * 8, 256, 0, st>>>(static_cast<const uint4*>(src), bytes / 16, sink);
    return cudaGetLastError();
}

cudaError_t launch_probe_tma(const void* src, size_t bytes, unsigned* status, cudaStream_t st) {
    static bool configured = false;
    const int smem = PROBE_CHUNK * PROBE_STAGES;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(probe_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    probe_tma_kernel<<<current_sm_count(), 32, smem, st>>>(static_cast<const uint8_t*>(src), bytes / PROBE_CHUNK, status);
    return cudaGetLastError();
}

cudaError_t launch_l2_flush(void* buf, size_t bytes, cudaStream_t st) {
    const size_t n16 = bytes / 16;
    if (!n16) return cudaSuccess;
    l2_flush_kernel<<<(unsigned)current_sm_count() * 8u, 256, 0, st>>>(static_cast<uint4*>(buf), n16);
    return cudaGetLastError();
}

}  // namespace nnb
