// MoE routing, dispatch and combine around the grouped W4A16 GEMM.
//
// Follows the reference's resident-expert path (crates/backend-gpu/src/rawcuda/w4a16_dec/moe/mod.rs:263-447,
// crates/backend-gpu/src/rawcuda/w4a16_dec/kernels/marlin_moe.rs:290-422):
//   router top-k -> group the T*k (token, expert) slots by expert -> grouped GEMM-1 over gate|up ->
//   SiLU(gate)*up -> grouped GEMM-2 over down, scaled by the routing weight -> sum over k.
// Kernels here: top-k (crates/backend-gpu/src/rawcuda/assets/moe.cu:686-759), the expert histogram / offsets /
// placement that replace the single-block counting sort (crates/backend-gpu/src/rawcuda/assets/gptq4.cu:376-413,
// crates/backend-gpu/src/rawcuda/assets/moe.cu:1599-1633), the row gather and the top-k sum
// (crates/backend-gpu/src/rawcuda/assets/moe.cu:1662-1674); the activation (:1649-1660) is in the first matmul's epilogue.
// Slots of one expert are placed in the order in which they were counted, so their order inside an expert's segment is
// not fixed; every output row is computed independently and the final sum runs over k in index order,
// so results do not depend on that order.
#include <cuda_fp16.h>

#include "dec.h"
#include "moe_topk.cuh"

namespace w4 {

namespace {

// Start of every kernel here.  They are small, and between two calls' matmuls their launches cost as much as their work: so they are
// launched with programmatic stream serialization, let the next kernel come as soon as they run, and touch nothing before the kernel
// before them is complete.  (In an ordinary launch both instructions do nothing.)
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr int TOPK_WARPS = 8;

// Rows per tile of an expert with c rows: `bm` of them, or (`even`) equal shares of at most bm, in multiples of 16 rows.
__device__ __forceinline__ int tile_step(int c, int bm, int even) {
    if (!even || c <= 0) {
        return bm;
    }
    const int nt = (c + bm - 1) / bm;
    return ((c + nt - 1) / nt + 15) & ~15;
}

// `cnt` (optional): rows per local expert, MOE_CNT_STRIDE apart; zero on entry, moe_offsets_kernel leaves it so.  What a slot's count was before
// it is its place in the expert's segment (`rank`): the gather asks for no place of its own.
// What bounds it at a prefill's sizes is the counting: 32768 atomics on 128 neighbouring words queued up in four lines of L2.  A sector for every
// counter and no second pass of atomics: layers of 512 tokens 124.9 -> 120.8 us, of 4096 354 -> 347 (with the sums below).
__global__ void moe_topk_kernel(const float* lg, int* idx, float* wt, int t, int n, int k, int stage_rows, int* cnt, int* rank, int e0, int e1) {
    extern __shared__ __align__(16) float s_stage[];   // [warps][n] when the launch provides it
    pdl_begin();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ti = blockIdx.x * TOPK_WARPS + w;
    if (ti >= t) {
        return;
    }
    const int e = topk_of_token(lg + (size_t)ti * n, idx + (size_t)ti * k, wt + (size_t)ti * k, n, k, lane,
                                stage_rows ? s_stage + (size_t)w * n : nullptr);
    if (cnt != nullptr && lane < k && e >= e0 && e < e1) {               // k <= 32
        rank[(size_t)ti * k + lane] = atomicAdd(cnt + e * MOE_CNT_STRIDE, 1);
    }
}

// Inclusive scan of (rows, tiles) over the block's 1024 threads: shuffles inside a warp, then the 32 warp totals.
__device__ __forceinline__ void scan_rows_tiles(int& vr, int& vt, int& total_rows, int& total_tiles, int* s_r, int* s_t) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int r = __shfl_up_sync(0xffffffffu, vr, d), tt = __shfl_up_sync(0xffffffffu, vt, d);
        if (lane >= d) {
            vr += r;
            vt += tt;
        }
    }
    if (lane == 31) {
        s_r[w] = vr;
        s_t[w] = vt;
    }
    __syncthreads();
    if (w == 0) {
        int tr = s_r[lane], tl = s_t[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int r = __shfl_up_sync(0xffffffffu, tr, d), tt = __shfl_up_sync(0xffffffffu, tl, d);
            if (lane >= d) {
                tr += r;
                tl += tt;
            }
        }
        s_r[lane] = tr;    // inclusive totals of warps 0..lane
        s_t[lane] = tl;
    }
    __syncthreads();
    if (w > 0) {
        vr += s_r[w - 1];
        vt += s_t[w - 1];
    }
    total_rows = s_r[31];
    total_tiles = s_t[31];
}

// Decode-sized batches (at most 1024 (token, expert) slots): routing, histogram, offsets, tile table, placement
// and sorted routing weights in ONE block of 1024 threads -- the launches they take otherwise cost more
// than the expert matmuls of a single token.  Same tables as the separate kernels below.
__global__ void __launch_bounds__(1024)
moe_route_small_kernel(const float* lg, int* idx, float* wt,
                       int* off, int* pos_of_slot, int* slot_of_pos,
                       int* tile_expert, int* tile_row0, int* tile_rows,
                       int* n_tiles, int* n_rows, float* row_w, int t, int n_exp,
                       int k, int e0, int e1, int bm, int stage_rows, int do_topk) {
    __shared__ int s_rows[1024], s_off[1024], s_cursor[1024], s_wr[32], s_wt[32], s_idx[8 * 32];
    extern __shared__ __align__(16) float s_stage[];   // [32 warps][n_exp] when the launch provides it
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    s_rows[tid] = 0;
    s_cursor[tid] = 0;
    pdl_begin();
    if (do_topk) {   // a handful of tokens: routed here; more: routed by moe_topk_kernel on many SMs just before
        for (int ti = w; ti < t; ti += 32) {
            const int e = topk_of_token(lg + (size_t)ti * n_exp, idx + (size_t)ti * k, wt + (size_t)ti * k, n_exp, k, lane,
                                        stage_rows ? s_stage + (size_t)w * n_exp : nullptr);
            if (lane < k) {
                s_idx[ti * k + lane] = e;                                // t <= 8, k <= 32
            }
        }
    }
    __syncthreads();   // idx / wt of every token are visible to the block
    const int ns = t * k;
    int my_e = -1;
    if (tid < ns) {
        my_e = do_topk ? s_idx[tid] : idx[tid];
        if (my_e >= e0 && my_e < e1) {
            atomicAdd(&s_rows[my_e], 1);
        } else {
            my_e = -1;
        }
    }
    __syncthreads();
    const int c = s_rows[tid];
    const int ct = (c + bm - 1) / bm;
    int vr = c, vt = ct, total_rows, total_tiles;
    scan_rows_tiles(vr, vt, total_rows, total_tiles, s_wr, s_wt);
    const int row0 = vr - c, tile0 = vt - ct;
    s_off[tid] = row0;
    if (tid < n_exp) {
        off[tid] = row0;
    }
    for (int r = 0, i = tile0; r < c; r += bm, ++i) {
        tile_expert[i] = tid;
        tile_row0[i] = row0 + r;
        tile_rows[i] = min(bm, c - r);
    }
    if (tid == 1023) {
        *n_tiles = total_tiles;
        *n_rows = total_rows;
    }
    __syncthreads();
    if (tid < ns) {
        int pos = -1;
        if (my_e >= 0) {
            pos = s_off[my_e] + atomicAdd(&s_cursor[my_e], 1);
            slot_of_pos[pos] = tid;
            row_w[pos] = wt[tid];
        }
        pos_of_slot[tid] = pos;  // -1: the expert lives on another rank
    }
}

// How an expert's rows are cut into tiles: of bm rows with a remainder, in equal shares of at most bm (multiples of 16), or like the first
// but with the table sorted.  Persistent CTAs take tiles in turn: sorted, no CTA gets more of the large ones than another.
// One block of 1024 threads (n_exp <= 1024): exclusive offsets of the local experts' segments and the m-tile
// table of the grouped GEMM, tile i -> (expert, first sorted row, valid rows).  Also clears the counts.
__global__ void __launch_bounds__(1024)
moe_offsets_kernel(int* cnt, int* off, int* tile_expert, int* tile_row0, int* tile_rows, int* n_tiles, int* n_rows,
                   int n_exp, int e0, int e1, int bm, int shares) {
    __shared__ int s_r[32], s_t[32];
    __shared__ __align__(16) int s_rest[1024];
    const int e = threadIdx.x;
    pdl_begin();
    const int c = (e >= e0 && e < e1) ? cnt[e * MOE_CNT_STRIDE] : 0;
    const int step = tile_step(c, bm, shares == TILES_EVEN), rest = shares == TILES_SORTED ? c % bm : 0;
    const int ct = shares == TILES_SORTED ? c / bm : (c + step - 1) / step;
    int vr = c, vt = ct, total_rows, total_tiles;
    scan_rows_tiles(vr, vt, total_rows, total_tiles, s_r, s_t);
    const int row0 = vr - c, tile0 = vt - ct;
    if (shares == TILES_SORTED) {
        // whole tiles first, then what is left of each expert, the largest first
        s_rest[e] = rest;
        const int rests = __syncthreads_count(rest > 0);
        if (rest > 0) {
            int rank = 0;
            for (int o = 0; o < n_exp; o += 4) {                     // (nothing is left of experts past the last)
                const int4 r4 = *reinterpret_cast<const int4*>(s_rest + o);
                rank += (r4.x > rest || (r4.x == rest && o < e)) + (r4.y > rest || (r4.y == rest && o + 1 < e)) +
                        (r4.z > rest || (r4.z == rest && o + 2 < e)) + (r4.w > rest || (r4.w == rest && o + 3 < e));
            }
            tile_expert[total_tiles + rank] = e;
            tile_row0[total_tiles + rank] = row0 + c - rest;
            tile_rows[total_tiles + rank] = rest;
        }
        total_tiles += rests;
    }
    if (e < n_exp) {
        off[e] = row0;
        cnt[e * MOE_CNT_STRIDE] = 0;
    }
    for (int r = 0, i = tile0; r < c - rest; r += step, ++i) {
        tile_expert[i] = e;
        tile_row0[i] = row0 + r;
        tile_rows[i] = min(step, c - r);
    }
    if (e == 1023) {
        *n_tiles = total_tiles;
        *n_rows = total_rows;
    }
}

// Placement of the local experts' slots in sorted order, with the routing weight of each sorted row (grouped matmul 2 multiplies by
// it), and xs[pos][:] = x[token][:] for the token's k slots (f16 rows of h).  A block takes a token: its first warp places the slots, then
// every thread reads 16 bytes of the row once and writes them to all of the token's places: bound by the writes (4096 tokens x 8 slots x
// 4 KB, cold: 39 us with a thread per 16 bytes of a slot, 33 with a warp per token, 31 so).
constexpr int GATHER_THREADS = 128;
__global__ void __launch_bounds__(GATHER_THREADS)
moe_place_gather_kernel(const uint4* x, uint4* xs, const int* idx, const float* wt, const int* off, int* pos_of_slot,
                        int* slot_of_pos, float* row_w, int t, int k, int h8, int e0, int e1) {
    __shared__ int s_pos[32];                                                        // k <= 32
    pdl_begin();
    for (int tok = (int)blockIdx.x; tok < t; tok += (int)gridDim.x) {
        if ((int)threadIdx.x < k) {
            const int slot = tok * k + (int)threadIdx.x, e = idx[slot];
            int pos = -1;                                                            // the expert lives on another rank
            if (e >= e0 && e < e1) {
                pos = off[e] + pos_of_slot[slot];                                     // (its rank so far)
                slot_of_pos[pos] = slot;
                row_w[pos] = wt[slot];
            }
            pos_of_slot[slot] = pos;
            s_pos[threadIdx.x] = pos;
        }
        __syncthreads();
        for (int c = (int)threadIdx.x; c < h8; c += 2 * GATHER_THREADS) {
            const bool two = c + GATHER_THREADS < h8;
            const uint4 v0 = x[(size_t)tok * h8 + c], v1 = two ? x[(size_t)tok * h8 + c + GATHER_THREADS] : make_uint4(0, 0, 0, 0);
            for (int j = 0; j < k; ++j) {
                const int pos = s_pos[j];
                if (pos >= 0) {
                    xs[(size_t)pos * h8 + c] = v0;
                    if (two) {
                        xs[(size_t)pos * h8 + c + GATHER_THREADS] = v1;
                    }
                }
            }
        }
        __syncthreads();                                                             // s_pos is for the next token
    }
}

// out[t][c] = sum_j c2[pos(t*k+j)][c]  (routing weights were applied in GEMM-2's epilogue); slots whose
// expert is not local contribute nothing.  The rows of eight slots are on their way at once:
// a slot after the other, each took two trips to memory, about 2 us of a decode call (a layer of one token 22.8 -> 20.7 us, of eight 50.1 -> 47.3).
constexpr int COMBINE_AHEAD = 8;
template <bool OUT_F16>
__global__ void moe_combine_kernel(const __half* c2, void* out, const int* pos_of_slot,
                                   int t, int h, int k) {
    pdl_begin();
    const int h8 = h / 8;
    const size_t total = (size_t)t * h8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / h8), c = (int)(i % h8) * 8;
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int j0 = 0; j0 < k; j0 += COMBINE_AHEAD) {
            int pos[COMBINE_AHEAD];
            uint4 v[COMBINE_AHEAD];
#pragma unroll
            for (int j = 0; j < COMBINE_AHEAD; ++j) {
                pos[j] = j0 + j < k ? pos_of_slot[r * k + j0 + j] : -1;
            }
#pragma unroll
            for (int j = 0; j < COMBINE_AHEAD; ++j) {
                if (pos[j] >= 0) {
                    v[j] = *reinterpret_cast<const uint4*>(c2 + (size_t)pos[j] * h + c);
                }
            }
#pragma unroll
            for (int j = 0; j < COMBINE_AHEAD; ++j) {
                if (pos[j] >= 0) {
                    const __half2* vh = reinterpret_cast<const __half2*>(&v[j]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 f = __half22float2(vh[q]);
                        acc[2 * q] += f.x;
                        acc[2 * q + 1] += f.y;
                    }
                }
            }
        }
        if (OUT_F16) {
            uint4 ov;
            __half2* oh = reinterpret_cast<__half2*>(&ov);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                oh[q] = __floats2half2_rn(acc[2 * q], acc[2 * q + 1]);
            }
            *reinterpret_cast<uint4*>((__half*)out + (size_t)r * h + c) = ov;
        } else {
            float4* o = reinterpret_cast<float4*>((float*)out + (size_t)r * h + c);
            o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
            o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        }
    }
}

inline int blocks_for(size_t total, int threads) {
    size_t b = (total + threads - 1) / threads;
    if (b > 148 * 16) {
        b = 148 * 16;
    }
    return b < 1 ? 1 : (int)b;
}

}  // namespace

namespace {

template <class... P, class... A>
cudaError_t launch(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, int pdl, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace

cudaError_t launch_moe_topk(const float* logits, int* idx, float* wt, int t, int n_exp, int k, int* cnt, int* rank, int e0, int e1,
                            int pdl, cudaStream_t st) {
    const int stage = n_exp <= 512;   // 8 warps x 512 floats = 16 KB of shared memory at most
    return launch(moe_topk_kernel, (t + TOPK_WARPS - 1) / TOPK_WARPS, TOPK_WARPS * 32, stage ? TOPK_WARPS * n_exp * sizeof(float) : 0, st,
                  pdl, logits, idx, wt, t, n_exp, k, stage, cnt, rank, e0, e1);
}

// Up to eight tokens are routed by the table block itself (one launch); above that one block's 32 warps would route two or more tokens
// each in turn (27 us at 64 tokens), so the routing runs on many SMs first and the block only builds the tables.
cudaError_t launch_moe_route_small(const float* logits, const MoeBufs& b, int t, int n_exp, int k, int e0, int e1, int bm, int pdl,
                                   cudaStream_t st, unsigned long long& launched) {
    const int stage = n_exp <= 256;   // 32 warps x 256 floats = 32 KB beside the 12 KB of tables
    const int own_topk = t <= 8;
    cudaError_t e = cudaSuccess;
    if (!own_topk) {
        e = launch_moe_topk(logits, b.idx, b.wt, t, n_exp, k, nullptr, nullptr, 0, 0, pdl, st);
        launched += e == cudaSuccess;
    }
    if (e == cudaSuccess) {
        e = launch(moe_route_small_kernel, 1, 1024, (stage && own_topk) ? 32 * n_exp * sizeof(float) : 0, st, pdl, logits, b.idx, b.wt,
                   b.off, b.pos_of_slot, b.slot_of_pos, b.tile_expert, b.tile_row0, b.tile_rows, b.n_tiles, b.n_rows, b.row_w, t, n_exp, k,
                   e0, e1, bm, stage, own_topk);
        launched += e == cudaSuccess;
    }
    return e;
}

cudaError_t launch_moe_sort(const float* logits, const void* x, const MoeBufs& b, int t, int n_exp, int k, int h, int e0, int e1, int bm,
                            int shares, int pdl, cudaStream_t st, unsigned long long& launched) {
    cudaError_t e = launch_moe_topk(logits, b.idx, b.wt, t, n_exp, k, b.cnt, b.pos_of_slot, e0, e1, pdl, st);
    if (e != cudaSuccess) {
        return e;
    }
    ++launched;
    e = launch(moe_offsets_kernel, 1, 1024, 0, st, pdl, b.cnt, b.off, b.tile_expert, b.tile_row0, b.tile_rows, b.n_tiles, b.n_rows,
               n_exp, e0, e1, bm, shares);
    if (e != cudaSuccess) {
        return e;
    }
    ++launched;
    e = launch(moe_place_gather_kernel, blocks_for((size_t)t, 1), GATHER_THREADS, 0, st, pdl, (const uint4*)x, (uint4*)b.xs, b.idx, b.wt,
               b.off, b.pos_of_slot, b.slot_of_pos, b.row_w, t, k, h / 8, e0, e1);
    launched += e == cudaSuccess;
    return e;
}

cudaError_t launch_moe_combine(const MoeBufs& b, void* out, int t, int h, int k, int out_f16, int pdl, cudaStream_t st) {
    const int g = blocks_for((size_t)t * (h / 8), 256);
    return launch(out_f16 ? moe_combine_kernel<true> : moe_combine_kernel<false>, g, 256, 0, st, pdl, (const __half*)b.c2, out,
                  b.pos_of_slot, t, h, k);
}

}  // namespace w4
