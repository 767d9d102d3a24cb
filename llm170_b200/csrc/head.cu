// int8 lm-head: per-row quantiser and the GEMV  out[t][n] = (sum_k q[n][k] * x[t][k]) * scale[n].
//
// Takes the place of W4a16Dec::upload_head (crates/backend-gpu/src/rawcuda/w4a16_dec/upload.rs:1472-1569: host threads
// quantise the bf16 matrix) and of the FFMA kernels w4a16_gemv_i8 / w4a16_gemv_i8_t
// (crates/backend-gpu/src/rawcuda/assets/head.cu:100-225, one 64-thread block per output row, launched from
// crates/backend-gpu/src/rawcuda/w4a16_dec/kernels/gemv.rs:64-110).  The lm-head is the largest weight stream of a
// decode step after the layers (vocabulary x hidden bytes), so the kernel is built for HBM bandwidth:
//   * the quantiser runs on the device, row chunks at a time, with the reference's arithmetic (f32 absmax / 127,
//     IEEE division, round half away from zero, clamp to +-127): the stored values are bit-identical to the host recipe;
//     they are kept offset-binary (q + 128) so that one byte permute puts two of them into the mantissas of two f16;
//   * a warp owns 16 whole rows at a time while there is a block of 16 rows for every warp of the GPU; the blocks left after
//     that are spread over all SMs, K split over the warps that would idle.  Each lane streams 16 bytes
//     of row g and of row g+8 per 64 channels, expands them to exact f16 and feeds them as the 16-row operand of
//     mma.sync m16n8k16; the tokens (up to 8 per pass) are the columns;
//   * the activations are f32 in the reference.  They are staged once per CTA as TWO f16 planes, hi = f16(x) and
//     lo = f16((x - hi) * 2^11), multiplied separately and recombined in f32: the products with the exact integer
//     weights carry x to about 2^-22 instead of the 2^-11 a single f16 plane would keep.
// No wait on another CTA anywhere in this file.
#include <cuda_fp16.h>

#include <algorithm>
#include <string>

#include "../../include/w4a16_b200.h"
#include "dec.h"
#include "gemv_common.cuh"

namespace w4 {

namespace {

constexpr int HEAD_THREADS = 512;       // 16 warps
constexpr int HEAD_TOK = 8;             // tokens per pass (columns of the MMA)
constexpr int HEAD_XPAD = 16;           // bytes added to a token's row of f16 so that quarter-warps hit distinct banks

__device__ __forceinline__ float bf16_bits_to_f32(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }

// Resident layout: [16 rows][64 channels][rows g / g + 8][32 lanes][16 bytes].  Lane 4g + t of the GEMV multiplies row g and row g + 8 at
// channels 16t..16t+15 of a 64-channel step; its 16 bytes of either lie beside those of the other lanes, so that a warp reads two whole
// 512-byte lines per step and 16 rows of the matrix are one contiguous piece.
__host__ __device__ __forceinline__ size_t head_at(size_t row, int ch, int k) {
    const size_t tile = row / 16 * (size_t)(k / 64) + (size_t)(ch / 64);
    const int r = (int)(row % 16);
    return tile * 1024 + (size_t)((r >> 3) * 512 + ((r & 7) * 4 + ch % 64 / 16) * 16 + ch % 16);
}

// One block per row, row0 + blockIdx.x: absmax, scale, quantise.  w: bf16 [rows][k] (device staging), q: offset-binary bytes (head_at).
// Rows from `n` on fill the last 16: zeros.
__global__ void __launch_bounds__(256) head_quant_kernel(const uint16_t* __restrict__ w, uint8_t* __restrict__ q,
                                                         float* __restrict__ scale, int row0, int n, int k) {
    __shared__ float red[8];
    __shared__ float s_scale;
    const size_t row = (size_t)row0 + blockIdx.x;
    if (row >= (size_t)n) {
        for (int i = threadIdx.x; i < k; i += blockDim.x) {
            q[head_at(row, i, k)] = 128;
        }
        return;
    }
    const uint16_t* wr = w + (size_t)blockIdx.x * (size_t)k;
    float amax = 0.0f;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        amax = fmaxf(amax, fabsf(bf16_bits_to_f32(wr[i])));
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = amax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = red[0];
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i) {
            m = fmaxf(m, red[i]);
        }
        const float s = m > 0.0f ? __fdiv_rn(m, 127.0f) : 1.0f;
        s_scale = s;
        scale[row] = s;
    }
    __syncthreads();
    const float s = s_scale;
    for (int i = threadIdx.x; i < k; i += blockDim.x) {
        float v = roundf(__fdiv_rn(bf16_bits_to_f32(wr[i]), s));   // half away from zero, as f32::round
        v = fminf(fmaxf(v, -127.0f), 127.0f);
        q[head_at(row, i, k)] = (uint8_t)((int)v + 128);
    }
}

// two offset-binary bytes of `w` (selected by `sel`) -> half2 of the exact integers q = byte - 128
__device__ __forceinline__ uint32_t ob_pair_to_half2(uint32_t w, uint32_t sel) {
    const uint32_t h = __byte_perm(w, 0x64646464u, sel);   // 0x64xx = 1024 + byte
    uint32_t r;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(h), "r"(0x64806480u));   // - 1152
    return r;
}

// Rows of whole row blocks out of the resident order, offset-binary -> two's complement.  A block takes a row at a time.
__global__ void __launch_bounds__(256) head_untile_kernel(const uint8_t* __restrict__ q, uint4* __restrict__ rows, int n, int k) {
    for (int r = blockIdx.x; r < n; r += gridDim.x) {
        for (int c = threadIdx.x; c < k / 16; c += blockDim.x) {
            uint4 v = *reinterpret_cast<const uint4*>(q + head_at((size_t)r, c * 16, k));
            v.x ^= 0x80808080u;
            v.y ^= 0x80808080u;
            v.z ^= 0x80808080u;
            v.w ^= 0x80808080u;
            rows[(size_t)r * (k / 16) + c] = v;
        }
    }
}

struct HeadArgs {
    const uint8_t* q;
    const float* scale;
    const float* x;     // f32 [t][k], tokens [t0, t0 + tp) of it are this pass
    float* out;         // f32 [t][n]
    int n, k, t0, tp;
};

// D = 64-channel steps that a warp has on the way in its ring; 0: loads to registers, eight steps unrolled, for activations that leave no room
// for a ring of three (head_depth).
template <int D>
__global__ void __launch_bounds__(HEAD_THREADS, D > 0 ? 2 : 1) head_gemv_i8_kernel(const HeadArgs a) {
    extern __shared__ __align__(128) unsigned char hsm[];
    constexpr int WARPS = HEAD_THREADS / 32;
    __shared__ float4 s_part[WARPS * 32];
    const int k = a.k, tp = a.tp;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int nrb = (a.n + 15) / 16, nsteps = k / 64;
    // Whole rounds: a row block per warp.  The rest of the row blocks is dealt over all SMs and, where it leaves warps idle,
    // each block's K over several warps of its CTA: 151936 rows are 4.01 rounds, and the fifth one cost as much as the others.
    const int all_warps = gridDim.x * WARPS, rounds = nrb / all_warps;
    const int rest0 = rounds * all_warps, rest = nrb - rest0;
    const int per_cta = (rest + (int)gridDim.x - 1) / (int)gridDim.x;            // 0..WARPS
    int ways = WARPS;
    while (ways > 1 && ways * per_cta > WARPS) {
        ways >>= 1;
    }
    const int sub = warp / ways, part = warp - sub * ways;
    const int rb_rest = rest0 + sub * (int)gridDim.x + (int)blockIdx.x;
    const bool live = sub < per_cta && rb_rest < nrb;
    const int s0_rest = nsteps * part / ways, n_rest = live ? nsteps * (part + 1) / ways - s0_rest : 0;

    // ---- weights: a private ring of D steps of 1 KB, filled by asynchronous copies in the order of use, across row blocks.  Every lane
    // reads back what it copied itself, so the loop has no barrier.  (One token, calls back to back: 151936 x 2048 47.8 us, 151936 x 5120 114; with
    // loads to registers, eight steps unrolled, 61.7 and 134: a warp had nothing on the way while it multiplied.)
    const uint32_t ring = smem_u32(hsm) + (uint32_t)warp * (D * 1024u) + (uint32_t)lane * 16u;
    const unsigned char* fp = nullptr;
    int fr = -1, fleft = 0;                                                      // round being requested, steps left in it
    uint32_t fdst = 0;
    auto fetch = [&]() {
        if (D == 0) {
            return;
        }
        if (fleft == 0 && fr < rounds) {
            ++fr;
            const int rb = fr < rounds ? fr * all_warps + (int)blockIdx.x * WARPS + warp : rb_rest;
            fleft = fr < rounds ? nsteps : n_rest;
            fp = a.q + ((size_t)rb * nsteps + (fr < rounds ? 0 : s0_rest)) * 1024 + lane * 16;
        }
        if (fleft > 0) {
            cp_async_16(ring + fdst, fp);
            cp_async_16(ring + fdst + 512u, fp + 512);
            fp += 1024;
            --fleft;
        }
        cp_async_commit();
        if ((fdst += 1024u) == D * 1024u) {
            fdst = 0;
        }
    };
#pragma unroll
    for (int d = 0; d < D; ++d) {
        fetch();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");                           // the weights do not depend on the kernel before, x may

    const int xrow = k * 2 + HEAD_XPAD;                 // bytes of one token's f16 row
    unsigned char* xhi = hsm + WARPS * D * 1024;
    unsigned char* xlo = xhi + (size_t)tp * xrow;
    // stage the activations: hi = f16(x), lo = f16((x - hi) * 2^11)
    for (int i = threadIdx.x; i < tp * (k / 2); i += HEAD_THREADS) {
        const int tok = i / (k / 2), c = (i - tok * (k / 2)) * 2;
        const float2 v = *reinterpret_cast<const float2*>(a.x + (size_t)(a.t0 + tok) * k + c);
        const __half h0 = __float2half_rn(v.x), h1 = __float2half_rn(v.y);
        const __half l0 = __float2half_rn((v.x - __half2float(h0)) * 2048.0f);
        const __half l1 = __float2half_rn((v.y - __half2float(h1)) * 2048.0f);
        *reinterpret_cast<__half2*>(xhi + (size_t)tok * xrow + c * 2) = __halves2half2(h0, h1);
        *reinterpret_cast<__half2*>(xlo + (size_t)tok * xrow + c * 2) = __halves2half2(l0, l1);
    }
    __syncthreads();

    // lanes whose column of the MMA holds no token read token 0: their sums are never stored
    const uint32_t xh_l = smem_u32(xhi) + (uint32_t)((g < tp ? g : 0) * xrow + tq * 32), xl_l = xh_l + (uint32_t)(tp * xrow);
    uint32_t rsrc = 0;
    // sums of row block rb (with a ring: of the next one in it), steps [s0, s1): .x, .y = row g, tokens 2tq, 2tq + 1;  .z, .w = row g + 8
    auto multiply = [&](int rb, int s0, int s1) {
        float ch[4] = {0.f, 0.f, 0.f, 0.f}, cl[4] = {0.f, 0.f, 0.f, 0.f};
        const uint4* wp = reinterpret_cast<const uint4*>(a.q + (size_t)rb * nsteps * 1024) + lane;
#pragma unroll(D > 0 ? 1 : 8)
        for (int s = s0; s < s1; ++s) {
            uint4 w0, w1;
            if (D > 0) {
                cp_async_wait_group<(D > 0 ? D - 1 : 0)>();
                w0 = lds128(ring + rsrc);
                w1 = lds128(ring + rsrc + 512u);
                fetch();
                if ((rsrc += 1024u) == D * 1024u) {
                    rsrc = 0;
                }
            } else {
                w0 = __ldg(wp + s * 64);
                w1 = __ldg(wp + s * 64 + 32);
            }
            const uint32_t ww0[4] = {w0.x, w0.y, w0.z, w0.w}, ww1[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 bh = lds128(xh_l + (uint32_t)(s * 128 + h * 16)), bl = lds128(xl_l + (uint32_t)(s * 128 + h * 16));
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    // MMA j multiplies the lane's channels 4j..4j+3: the k order inside the MMA is permuted the same way
                    // for the weights and for the activations, which leaves every product in place
                    const int j = 2 * h + i;
                    uint32_t af[4];
                    af[0] = ob_pair_to_half2(ww0[j], 0x4140u);
                    af[1] = ob_pair_to_half2(ww1[j], 0x4140u);
                    af[2] = ob_pair_to_half2(ww0[j], 0x4342u);
                    af[3] = ob_pair_to_half2(ww1[j], 0x4342u);
                    mma16816(ch, af, i ? bh.z : bh.x, i ? bh.w : bh.y);
                    mma16816(cl, af, i ? bl.z : bl.x, i ? bl.w : bl.y);
                }
            }
        }
        return make_float4(ch[0] + cl[0] * (1.0f / 2048.0f), ch[1] + cl[1] * (1.0f / 2048.0f), ch[2] + cl[2] * (1.0f / 2048.0f),
                           ch[3] + cl[3] * (1.0f / 2048.0f));
    };
    auto store = [&](int rb, const float4& c) {
        const int ra = rb * 16 + g, rbb = ra + 8;
        const float sa = ra < a.n ? a.scale[ra] : 0.f, sb = rbb < a.n ? a.scale[rbb] : 0.f;
        const float ca[2] = {c.x, c.y}, cb[2] = {c.z, c.w};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int tok = 2 * tq + i;
            if (tok < tp) {
                float* o = a.out + (size_t)(a.t0 + tok) * a.n;
                if (ra < a.n) {
                    o[ra] = ca[i] * sa;
                }
                if (rbb < a.n) {
                    o[rbb] = cb[i] * sb;
                }
            }
        }
    };
    for (int i = 0; i < rounds; ++i) {
        const int rb = i * all_warps + (int)blockIdx.x * WARPS + warp;
        store(rb, multiply(rb, 0, nsteps));
    }
    if (rest == 0) {
        return;
    }
    float4 c = multiply(rb_rest, s0_rest, s0_rest + n_rest);
    if (ways > 1) {
        s_part[threadIdx.x] = c;
        __syncthreads();
        if (part == 0) {
            for (int w = 1; w < ways; ++w) {                                     // in K order
                const float4 o = s_part[threadIdx.x + w * 32];
                c.x += o.x;
                c.y += o.y;
                c.z += o.z;
                c.w += o.w;
            }
        }
    }
    if (live && part == 0) {
        store(rb_rest, c);
    }
}

constexpr int HEAD_DEPTHS[] = {8, 6, 5, 4, 3, 0};
constexpr size_t HEAD_SMEM_MAX = 218 * 1024;            // beside 8 KB for the sums
// Steps on the way per warp beside `x_bytes` of activations: five where that leaves room for a second CTA (the next call's, whose weights
// are then on the way before this one ends), else what fits beside them.
int head_depth(size_t x_bytes) {
    if (x_bytes + 5 * (HEAD_THREADS / 32 * 1024) <= (size_t)104 * 1024) {
        return 5;
    }
    for (int d : HEAD_DEPTHS) {
        if (x_bytes + (size_t)d * (HEAD_THREADS / 32 * 1024) <= HEAD_SMEM_MAX) {
            return d;
        }
    }
    return 0;
}
const void* head_kernel(int depth) {
    switch (depth) {
    case 8: return (const void*)head_gemv_i8_kernel<8>;
    case 6: return (const void*)head_gemv_i8_kernel<6>;
    case 5: return (const void*)head_gemv_i8_kernel<5>;
    case 4: return (const void*)head_gemv_i8_kernel<4>;
    case 3: return (const void*)head_gemv_i8_kernel<3>;
    default: return (const void*)head_gemv_i8_kernel<0>;
    }
}

}  // namespace

cudaError_t head_init_device() {
    for (int d : HEAD_DEPTHS) {
        const cudaError_t e = cudaFuncSetAttribute(head_kernel(d), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HEAD_SMEM_MAX);
        if (e != cudaSuccess) {
            return e;
        }
    }
    return cudaSuccess;
}

}  // namespace w4

using w4::Dec;

extern "C" {

int w4a16_upload_head(w4a16_dec* dec, const void* w_bf16_host, size_t bytes, int n, int k) {
    Dec& d = dec->d;
    if (n < 1 || k < 64 || k % 64 != 0 || w_bf16_host == nullptr || bytes < (size_t)n * k * 2) {
        return d.fail("w4a16 upload_head: shape contract n=%d k=%d (k a multiple of 64) bytes=%zu", n, k, bytes);
    }
    if ((size_t)w4::HEAD_XPAD + (size_t)k * 2 > (size_t)100 * 1024) {
        return d.fail("w4a16 upload_head: k=%d: one token's two f16 planes do not fit in shared memory", k);
    }
    cudaSetDevice(d.device);
    cudaDeviceSynchronize();
    if (d.head_q) {
        d.retired.push_back(d.head_q);      // a captured graph may still name them
        d.retired.push_back(d.head_scale);
        d.weights_bytes -= (size_t)d.head_n * d.head_k + (size_t)d.head_n * 4;
        d.head_q = nullptr;
        d.head_scale = nullptr;
        d.head_n = d.head_k = 0;
    }
    uint8_t* q = nullptr;
    float* sc = nullptr;
    uint16_t* stage = nullptr;
    const int rows_chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)n, ((size_t)32 << 20) / ((size_t)k * 2)));
    const int n16 = (n + 15) / 16 * 16;
    cudaError_t e = cudaMalloc(&q, (size_t)n16 * k);
    if (e == cudaSuccess) e = cudaMalloc(&sc, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&stage, (size_t)rows_chunk * k * 2);
    if (e != cudaSuccess) {
        cudaFree(q);
        cudaFree(sc);
        cudaFree(stage);
        return d.cuda_fail("alloc lm-head", e);
    }
    for (int r0 = 0; r0 < n && e == cudaSuccess; r0 += rows_chunk) {
        const int rows = std::min(rows_chunk, n - r0);
        e = cudaMemcpyAsync(stage, (const unsigned char*)w_bf16_host + (size_t)r0 * k * 2, (size_t)rows * k * 2,
                            cudaMemcpyHostToDevice, d.stream);
        if (e == cudaSuccess) {
            w4::head_quant_kernel<<<r0 + rows == n ? n16 - r0 : rows, 256, 0, d.stream>>>(stage, q, sc, r0, n, k);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            e = cudaStreamSynchronize(d.stream);   // the staging chunk is reused
        }
    }
    cudaFree(stage);
    if (e != cudaSuccess) {
        cudaFree(q);
        cudaFree(sc);
        return d.cuda_fail("quantise lm-head", e);
    }
    d.head_q = q;
    d.head_scale = sc;
    d.head_n = n;
    d.head_k = k;
    d.weights_bytes += (size_t)n * k + (size_t)n * 4;
    return 0;
}

int w4a16_head_spec(w4a16_dec* dec, int* n, int* k) {
    Dec& d = dec->d;
    if (!d.head_q) {
        return d.fail("w4a16 head: no lm-head uploaded");
    }
    if (n) *n = d.head_n;
    if (k) *k = d.head_k;
    return 0;
}

int w4a16_head_unpack(w4a16_dec* dec, void* q_host, void* scale_host) {
    Dec& d = dec->d;
    if (!d.head_q) {
        return d.fail("w4a16 head: no lm-head uploaded");
    }
    cudaSetDevice(d.device);
    // 32 MB of whole row blocks at a time (less where the device has no room), from the resident order to rows on the device
    const int k = d.head_k;
    int rows_chunk = (int)std::min<size_t>(std::max<size_t>(16, ((size_t)32 << 20) / k / 16 * 16), (size_t)(d.head_n + 15) / 16 * 16);
    uint4* rows_dev = nullptr;
    cudaError_t e = cudaMalloc(&rows_dev, (size_t)rows_chunk * k);
    while (e != cudaSuccess && rows_chunk > 16) {
        cudaGetLastError();
        rows_chunk = std::max(16, rows_chunk / 2 / 16 * 16);
        e = cudaMalloc(&rows_dev, (size_t)rows_chunk * k);
    }
    for (int r0 = 0; r0 < d.head_n && e == cudaSuccess; r0 += rows_chunk) {
        const int rows = std::min(rows_chunk, d.head_n - r0);
        w4::head_untile_kernel<<<std::min(rows, 148 * 16), 256, 0, d.stream>>>(d.head_q + (size_t)r0 * k, rows_dev, rows, k);
        e = cudaGetLastError();
        if (e == cudaSuccess) {
            e = cudaMemcpyAsync((unsigned char*)q_host + (size_t)r0 * k, rows_dev, (size_t)rows * k, cudaMemcpyDeviceToHost, d.stream);
        }
        if (e == cudaSuccess) {
            e = cudaStreamSynchronize(d.stream);
        }
    }
    cudaFree(rows_dev);
    if (e == cudaSuccess && scale_host) {
        e = cudaMemcpy(scale_host, d.head_scale, (size_t)d.head_n * 4, cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) {
        return d.cuda_fail("read lm-head", e);
    }
    return 0;
}

int w4a16_head_forward(w4a16_dec* dec, const float* x32_dev, float* out_dev, int t, void* stream) {
    Dec& d = dec->d;
    if (!d.head_q) {
        return d.fail("w4a16 head_forward: no lm-head uploaded");
    }
    if (t < 1 || t > 16) {
        return d.fail("w4a16 head_forward: t=%d, must be 1..16", t);   // the reference's limit (assets/head.cu:159)
    }
    if (((uintptr_t)x32_dev & 7) != 0 || ((uintptr_t)out_dev & 3) != 0) {
        return d.fail("w4a16 head_forward: x must be 8-byte aligned and out 4-byte aligned");
    }
    cudaStream_t st = stream ? (cudaStream_t)stream : d.stream;
    const size_t xrow = (size_t)d.head_k * 2 + w4::HEAD_XPAD;
    const int tp_max = (int)std::min<size_t>(w4::HEAD_TOK, ((size_t)200 * 1024) / (2 * xrow));
    const int nrb = (d.head_n + 15) / 16;
    const int grid = std::min(d.sm_count, nrb);
    for (int t0 = 0; t0 < t; t0 += tp_max) {
        w4::HeadArgs a;
        a.q = d.head_q;
        a.scale = d.head_scale;
        a.x = x32_dev;
        a.out = out_dev;
        a.n = d.head_n;
        a.k = d.head_k;
        a.t0 = t0;
        a.tp = std::min(tp_max, t - t0);
        const int depth = w4::head_depth(2 * (size_t)a.tp * xrow);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(w4::HEAD_THREADS);
        cfg.dynamicSmemBytes = 2 * (size_t)a.tp * xrow + (size_t)depth * (w4::HEAD_THREADS / 32 * 1024);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        if (d.tune_pdl) {
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
        }
        void* args[] = {&a};
        cudaError_t e = cudaLaunchKernelExC(&cfg, w4::head_kernel(depth), args);
        if (e != cudaSuccess) {
            return d.cuda_fail("launch lm-head gemv", e);
        }
        d.launches++;
    }
    d.last_kernel = "head_gemv_i8_kernel";
    return 0;
}

}  // extern "C"
