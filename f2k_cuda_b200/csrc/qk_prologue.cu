// Memory-bound kernels in front of the attention: per-head RMSNorm and 4-axis RoPE.
//
//  * qk_prologue_kernel     both steps fused, for the Q and K of up to two streams in
//                           ONE launch: reads each raw element once, writes the
//                           normalised + rotated bf16 once (one rounding instead of the
//                           reference's two). Replaces, per block, the reference's
//                           2-4 rmsnorm_bf16 launches, 2-4 rope_4axis_inplace_bf16
//                           launches and the fill_pos_ids_expanded launches
//                           (F2K_CUDA src/backend/cuda/double_stream_block.cu:290-372,
//                           single_stream_block.cu:254-264).
//  * rmsnorm_rows_kernel*   stand-alone RMSNorm with the reference's contract
//                           (src/backend/cuda/kernels/rmsnorm.cu:42-88).
//  * rope4_rows_kernel*     stand-alone interleaved-pair rotation with the reference's
//                           contract (src/backend/cuda/kernels/rope_4axis.cu:13-54).
//
// All of them are HBM-bound: 16-byte loads/stores, a half-warp (dim 128) or a warp per
// 128-element head row, grid sized as a multiple of the SM count, grid-stride loop.
//
// The head_dim 128 kernels may start while the kernel in front of them still runs and writes what they
// read, whatever it is: rows, gains, tables or positions. So they read with plain loads only, behind
// griddepcontrol.wait: __ldg and `const __restrict__` promise that nobody writes the data for as long as the
// kernel lives, and plain `__restrict__` that the wait does not touch it; either lets a load move ahead of it.

#include "attn_launch.h"
#include "row_math.cuh"

#include <cuda_bf16.h>

namespace f2k {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ float warp_sum(float v) {
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 16);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 8);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 4);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    return v;
}

// ---------------------------------------------------------------------------------
// Fused RMSNorm + RoPE, head_dim 128. A half-warp owns one head row: lane i holds
// elements [8i, 8i+8) = rotation pairs 4i .. 4i+3, so both the reduction and the
// rotation stay inside the half-warp and inside a lane respectively.
// ---------------------------------------------------------------------------------
// A half-warp takes kGroup consecutive head rows of ONE token per iteration (kGroup divides the
// head count): their loads are issued back to back (kGroup x 16 bytes in flight per lane), and the
// token's table row and the gains are fetched once for the group.
template <int kGroup>
__global__ void __launch_bounds__(kBlock, 4)
qk_prologue_kernel(const __grid_constant__ QkPrologueParams p) {
    // The attention kernel behind this one may set itself up while this one drains; and this one may
    // have started before the kernel in front of it has ended.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int hl = threadIdx.x & 15;  // lane inside the half-warp
    // Row numbers fit 32 bits (2^31 rows of 256 bytes exceed any memory; the launch checks it): two
    // 64-bit divisions per group of rows took more instructions than the arithmetic.
    const unsigned total = (unsigned)p.row_start[p.n_jobs] / kGroup;          // in groups
    const unsigned n_hw  = gridDim.x * (kBlock / 16);
    for (unsigned grp = blockIdx.x * (kBlock / 16) + (threadIdx.x >> 4); grp < total; grp += n_hw) {
        const unsigned row = grp * kGroup;
        int j = 0;
#pragma unroll
        for (int i = 1; i < kMaxPrologueJobs; ++i)
            if (i < p.n_jobs && row >= (unsigned)p.row_start[i]) j = i;
        const QkPrologueJob& job = p.job[j];
        const unsigned lr = row - (unsigned)p.row_start[j];
        const unsigned trow = lr / (unsigned)p.n_heads;         // token row over batch * seq
        const unsigned tok = trow % (unsigned)job.seq;
        const unsigned hd0 = lr - trow * (unsigned)p.n_heads;   // first head of the group
        // A token row of x may be a slice of a wider row (x_tok_stride); y is always dense.
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(job.x) +
                                                          (long long)trow * job.x_tok_stride + hd0 * kHeadDim);
        uint4 raw[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) raw[u] = src[u * 16 + hl];
        const uint4  graw = reinterpret_cast<const uint4*>(job.gamma)[hl];
        const float4 c4 = reinterpret_cast<const float4*>(job.cos_tab + (long long)tok * 64)[hl];
        const float4 s4 = reinterpret_cast<const float4*>(job.sin_tab + (long long)tok * 64)[hl];
        float g[8];
        unpack8(graw, g);
        const float cs[4] = {c4.x, c4.y, c4.z, c4.w};
        const float sn[4] = {s4.x, s4.y, s4.z, s4.w};
        uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(job.y) + (long long)lr * kHeadDim);
#pragma unroll
        for (int u = 0; u < kGroup; ++u) dst[u * 16 + hl] = norm_rope_row(raw[u], g, cs, sn, p.eps);
    }
}

// ---------------------------------------------------------------------------------
// Head exchange: the same row arithmetic, every row stored into the memory of the rank that owns
// its head (peer stores over NVLink, 256 contiguous bytes per half-warp and row). Work item =
// kGroup consecutive heads (all of one destination) of one token of one of the three tensors.
// ---------------------------------------------------------------------------------
template <int kGroup>
__global__ void __launch_bounds__(kBlock, 4)
qkv_scatter_kernel(const __grid_constant__ QkvScatterParams p) {
    const int hl = threadIdx.x & 15;
    const long long per_tensor = (long long)p.s_loc * p.n_heads / kGroup;
    const long long total = 3 * per_tensor;
    const long long n_hw  = (long long)gridDim.x * (kBlock / 16);
    for (long long grp = (long long)blockIdx.x * (kBlock / 16) + (threadIdx.x >> 4); grp < total; grp += n_hw) {
        const int which = (int)(grp / per_tensor);                       // 0 q, 1 k, 2 v
        const long long lr = (grp - which * per_tensor) * kGroup;        // row inside the tensor
        const int tok = (int)(lr / p.n_heads);
        const int hd0 = (int)(lr - (long long)tok * p.n_heads);
        const int dst_rank = hd0 / p.heads_per_rank;
        const int hh = hd0 - dst_rank * p.heads_per_rank;
        const void* xin = which == 0 ? p.q : (which == 1 ? p.k : p.v);
        unsigned char* base = which == 0 ? p.dst_q[dst_rank] : (which == 1 ? p.dst_k[dst_rank] : p.dst_v[dst_rank]);
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(xin) + lr * kHeadDim);
        uint4* dst = reinterpret_cast<uint4*>(
            base + (((long long)p.rank * p.s_loc + tok) * p.heads_per_rank + hh) * (long long)(kHeadDim * 2));
        uint4 raw[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) raw[u] = src[u * 16 + hl];
        if (which == 2) {
#pragma unroll
            for (int u = 0; u < kGroup; ++u) dst[u * 16 + hl] = raw[u];
            continue;
        }
        const uint4  graw = __ldg(reinterpret_cast<const uint4*>(which == 0 ? p.gamma_q : p.gamma_k) + hl);
        const float4 c4 = __ldg(reinterpret_cast<const float4*>(p.cos_tab + (long long)tok * 64) + hl);
        const float4 s4 = __ldg(reinterpret_cast<const float4*>(p.sin_tab + (long long)tok * 64) + hl);
        float g[8];
        unpack8(graw, g);
        const float cs[4] = {c4.x, c4.y, c4.z, c4.w};
        const float sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            float v[8];
            unpack8(raw[u], v);
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
            ss = half_warp_sum(ss);
            const float rrms = rsqrtf(ss * (1.0f / kHeadDim) + p.eps);
            float y[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float a = v[2 * k] * rrms * g[2 * k];
                const float b = v[2 * k + 1] * rrms * g[2 * k + 1];
                rotate_pair(y[2 * k], y[2 * k + 1], a, b, cs[k], sn[k]);
            }
            dst[u * 16 + hl] = pack8(y);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // the same publication as f2k::ptx::grid_done_publish, spelled out here to keep this file
        // free of the PTX header
        __threadfence_system();
        const unsigned int seen = atomicAdd(p.counter, 1u);
        if (seen == gridDim.x - 1u) {
            atomicExch(p.counter, 0u);
            __threadfence_system();
            for (int i = 0; i < p.world; ++i)
                asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.flag[i]), "r"(p.value) : "memory");
        }
    }
}

// ---------------------------------------------------------------------------------
// Stand-alone RMSNorm. dim == 128: half-warp per row, one pass. Other dims (multiple
// of 8): one warp per row, two passes over the row (the second hits L1/L2).
// A half-warp takes kRowsAhead consecutive rows at a time, their loads issued back to back (see
// rows_ahead): with many rows, one at a time is bound by the latency of one 16-byte load per lane.
// y = bf16( x * rsqrt(mean(x^2) + eps) * gamma ), fp32 arithmetic.
// ---------------------------------------------------------------------------------
template <int kRowsAhead>
__global__ void __launch_bounds__(kBlock)
rmsnorm_rows128_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma,
                       __nv_bfloat16* y, long long rows, float eps) {  // y may alias x
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int hl = threadIdx.x & 15;
    const long long n_hw = (long long)gridDim.x * (kBlock / 16);
    const uint4 graw = reinterpret_cast<const uint4*>(gamma)[hl];
    float g[8];
    unpack8(graw, g);
    for (long long row0 = ((long long)blockIdx.x * (kBlock / 16) + (threadIdx.x >> 4)) * kRowsAhead; row0 < rows;
         row0 += n_hw * kRowsAhead) {
        uint4 raw[kRowsAhead];
#pragma unroll
        for (int u = 0; u < kRowsAhead; ++u)
            if (row0 + u < rows) raw[u] = reinterpret_cast<const uint4*>(x + (row0 + u) * 128)[hl];
#pragma unroll
        for (int u = 0; u < kRowsAhead; ++u) {
            if (row0 + u >= rows) break;                     // the same for the whole half-warp
            float v[8];
            unpack8(raw[u], v);
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
            ss = half_warp_sum(ss);
            const float rrms = rsqrtf(ss * (1.0f / 128.0f) + eps);
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = v[i] * rrms * g[i];
            reinterpret_cast<uint4*>(y + (row0 + u) * 128)[hl] = pack8(o);
        }
    }
}

__global__ void __launch_bounds__(kBlock)
rmsnorm_rows_generic_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ gamma,
                            __nv_bfloat16* y, long long rows, int dim, float inv_dim,
                            float eps) {  // y may alias x
    const int lane = threadIdx.x & 31;
    const long long n_w = (long long)gridDim.x * (kBlock / 32);
    const int chunks = dim >> 3;  // 16-byte chunks per row
    for (long long row = (long long)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows;
         row += n_w) {
        const uint4* xr = reinterpret_cast<const uint4*>(x + row * dim);
        float ss = 0.f;
        for (int ch = lane; ch < chunks; ch += 32) {
            float v[8];
            unpack8(xr[ch], v);
#pragma unroll
            for (int i = 0; i < 8; ++i) ss = fmaf(v[i], v[i], ss);
        }
        ss = warp_sum(ss);
        const float rrms = rsqrtf(ss * inv_dim + eps);
        uint4* yr = reinterpret_cast<uint4*>(y + row * dim);
        for (int ch = lane; ch < chunks; ch += 32) {
            float v[8], g[8], o[8];
            unpack8(xr[ch], v);
            unpack8(__ldg(reinterpret_cast<const uint4*>(gamma) + ch), g);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = v[i] * rrms * g[i];
            yr[ch] = pack8(o);
        }
    }
}

// ---------------------------------------------------------------------------------
// Stand-alone rotation, in place. pos = clamp(pos_ids[row], 0, seq_max - 1);
// x'[2k] = x[2k] c - x[2k+1] s ; x'[2k+1] = x[2k] s + x[2k+1] c with c, s = table[pos][k].
// ---------------------------------------------------------------------------------
template <int kRowsAhead>
__global__ void __launch_bounds__(kBlock)
rope4_rows128_kernel(__nv_bfloat16* x, const float* cos_tab,
                     const float* sin_tab, const int32_t* pos_ids,
                     long long rows, int seq_max) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int hl = threadIdx.x & 15;
    const long long n_hw = (long long)gridDim.x * (kBlock / 16);
    for (long long row0 = ((long long)blockIdx.x * (kBlock / 16) + (threadIdx.x >> 4)) * kRowsAhead; row0 < rows;
         row0 += n_hw * kRowsAhead) {
        uint4 raw[kRowsAhead];
        int pos[kRowsAhead];
#pragma unroll
        for (int u = 0; u < kRowsAhead; ++u)
            if (row0 + u < rows) {
                raw[u] = reinterpret_cast<const uint4*>(x + (row0 + u) * 128)[hl];
                const int pid = pos_ids[row0 + u];
                pos[u] = pid >= seq_max ? seq_max - 1 : (pid < 0 ? 0 : pid);
            }
        float4 c4, s4;
#pragma unroll
        for (int u = 0; u < kRowsAhead; ++u) {
            if (row0 + u >= rows) break;
            if (u == 0 || pos[u] != pos[u - 1]) {            // the heads of one token share a table row
                c4 = reinterpret_cast<const float4*>(cos_tab + (long long)pos[u] * 64)[hl];
                s4 = reinterpret_cast<const float4*>(sin_tab + (long long)pos[u] * 64)[hl];
            }
            float v[8], o[8];
            unpack8(raw[u], v);
            const float cs[4] = {c4.x, c4.y, c4.z, c4.w};
            const float sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) rotate_pair(o[2 * k], o[2 * k + 1], v[2 * k], v[2 * k + 1], cs[k], sn[k]);
            reinterpret_cast<uint4*>(x + (row0 + u) * 128)[hl] = pack8(o);
        }
    }
}

__global__ void __launch_bounds__(kBlock)
rope4_rows_generic_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cos_tab,
                          const float* __restrict__ sin_tab, const int32_t* __restrict__ pos_ids,
                          long long rows, int head_dim, int seq_max) {
    const int lane = threadIdx.x & 31;
    const long long n_w = (long long)gridDim.x * (kBlock / 32);
    const int half = head_dim >> 1;
    for (long long row = (long long)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); row < rows;
         row += n_w) {
        int pos = __ldg(pos_ids + row);
        pos = pos >= seq_max ? seq_max - 1 : (pos < 0 ? 0 : pos);
        uint32_t* xr = reinterpret_cast<uint32_t*>(x + row * head_dim);
        const float* cr = cos_tab + (long long)pos * half;
        const float* sr = sin_tab + (long long)pos * half;
        for (int k = lane; k < half; k += 32) {
            const uint32_t w = xr[k];
            const float x0 = __uint_as_float(w << 16);
            const float x1 = __uint_as_float(w & 0xFFFF0000u);
            const float c = __ldg(cr + k), s = __ldg(sr + k);
            float y0, y1;
            rotate_pair(y0, y1, x0, x1, c, s);
            xr[k] = pack2(y0, y1);
        }
    }
}

int sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
    }();
    return sms;
}

constexpr int kBlocksPerSm = 8;  // 8 x 256 threads = a full SM of resident threads

int grid_for(long long units, int units_per_block) {
    const long long need = (units + units_per_block - 1) / units_per_block;
    const long long cap  = (long long)sm_count() * kBlocksPerSm;
    return (int)(need < cap ? (need > 0 ? need : 1) : cap);
}

// Rows a half-warp of the stand-alone kernels takes at a time. While the largest grid has a half-warp for every
// row, four at a time only leave blocks out: 300 rows rmsnorm / rope 1.39 / 1.37 us with one, 1.83 / 2.01 with
// four; 18432 rows 2.67 / 2.29 and 2.66 / 2.57. Beyond, the latency of one load per lane shows: 36864 rows
// 3.67 / 3.27 with one, 3.00 / 2.84 with four (launches back to back in a graph).
int rows_ahead(long long rows) { return rows <= (long long)sm_count() * kBlocksPerSm * (kBlock / 16) ? 1 : 4; }

// A launch that may start while the kernel in front of it drains; the kernel itself waits for that one's
// end before it touches memory.
template <typename... P, typename... A>
cudaError_t launch_overlapping(void (*kernel)(P...), int grid, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kBlock);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace

cudaError_t qk_prologue_prepare() {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, qk_prologue_kernel<4>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, qk_prologue_kernel<1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, qkv_scatter_kernel<4>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, qkv_scatter_kernel<1>);
    return e;
}

cudaError_t qk_prologue_launch(const QkPrologueParams& params, cudaStream_t stream) {
    QkPrologueParams p = params;
    for (int i = 0; i < p.n_jobs; ++i)
        if (p.job[i].x_tok_stride == 0) p.job[i].x_tok_stride = (long long)p.n_heads * kHeadDim;
    const long long total = p.row_start[p.n_jobs];
    if (total <= 0) return cudaSuccess;
    if (total >= 1ll << 31) return cudaErrorInvalidValue;
    if (p.n_heads % 4 == 0) return launch_overlapping(qk_prologue_kernel<4>, grid_for(total / 4, kBlock / 16), stream, p);
    return launch_overlapping(qk_prologue_kernel<1>, grid_for(total, kBlock / 16), stream, p);
}

cudaError_t qkv_scatter_launch(const QkvScatterParams& p, cudaStream_t stream) {
    const long long rows = 3ll * p.s_loc * p.n_heads;
    if (rows <= 0) return cudaErrorInvalidValue;
    if (p.heads_per_rank % 4 == 0)
        qkv_scatter_kernel<4><<<grid_for(rows / 4, kBlock / 16), kBlock, 0, stream>>>(p);
    else
        qkv_scatter_kernel<1><<<grid_for(rows, kBlock / 16), kBlock, 0, stream>>>(p);
    return cudaPeekAtLastError();
}

cudaError_t rmsnorm_rows_launch(const void* x, const void* gamma, void* y, int rows, int dim,
                                float eps, cudaStream_t stream) {
    auto xb = static_cast<const __nv_bfloat16*>(x);
    auto gb = static_cast<const __nv_bfloat16*>(gamma);
    auto yb = static_cast<__nv_bfloat16*>(y);
    if (dim == 128) {
        const int ahead = rows_ahead(rows);
        return launch_overlapping(ahead == 1 ? rmsnorm_rows128_kernel<1> : rmsnorm_rows128_kernel<4>,
                                  grid_for(rows, kBlock / 16 * ahead), stream, xb, gb, yb, (long long)rows, eps);
    } else {
        rmsnorm_rows_generic_kernel<<<grid_for(rows, kBlock / 32), kBlock, 0, stream>>>(
            xb, gb, yb, rows, dim, 1.0f / (float)dim, eps);
    }
    return cudaPeekAtLastError();
}

cudaError_t rope4_rows_launch(void* x, const float* cos_tab, const float* sin_tab,
                              const int32_t* pos_ids, int rows, int head_dim, int seq_max,
                              cudaStream_t stream) {
    auto xb = static_cast<__nv_bfloat16*>(x);
    if (head_dim == 128) {
        const int ahead = rows_ahead(rows);
        return launch_overlapping(ahead == 1 ? rope4_rows128_kernel<1> : rope4_rows128_kernel<4>,
                                  grid_for(rows, kBlock / 16 * ahead), stream, xb, cos_tab, sin_tab, pos_ids,
                                  (long long)rows, seq_max);
    } else {
        rope4_rows_generic_kernel<<<grid_for(rows, kBlock / 32), kBlock, 0, stream>>>(
            xb, cos_tab, sin_tab, pos_ids, rows, head_dim, seq_max);
    }
    return cudaPeekAtLastError();
}

}  // namespace f2k
