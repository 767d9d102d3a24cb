// Router top-k of a token by one warp, shared by the routing kernels (moe.cu) and by the matmuls that route themselves (gemv_moe_few.cu).
#pragma once
#include <cuda_runtime.h>

namespace w4 {

// One warp per token, experts dealt to lanes round-robin (expert e lives in lane e % 32, slot e / 32).
// Same arithmetic as select_topk / moe_topk of the reference (crates/core/src/qwen35/stages/moe.rs:8-31,
// crates/backend-gpu/src/rawcuda/w4a16_dec/mod.rs:168-185), in the same order: p_e = exp(l_e - max) / sum with the
// sum taken sequentially over e = 0..n-1, pick k times the largest remaining p (ties: lower index), weights =
// p / (sum of the picked p, added in pick order).  Ordering on the normalised p, not on the numerators, matters
// when two different numerators round to the same p.  exp is evaluated in double and rounded once, the closest
// a device routine gets to the host's expf.  A pick is two warp-wide integer reductions: positive floats order
// like their bit patterns, so the largest p is a max over u32 and the tie-break a min over the indices that hold it.
// `stage`: optional shared-memory row of n floats owned by this warp; with it the sequential sum is read back by one
// lane (independent loads, one dependent add each) instead of travelling through n dependent shuffles.
// SLOTS = experts per lane the instantiation can hold (n <= 32 * SLOTS): a compile-time bound keeps the lane's values in
// registers.
// Returns the lane's pick: lane r < k has the r-th one.
template <int SLOTS>
__device__ __forceinline__ int topk_of_token_n(const float* l, int* idx, float* wt,
                                               int n, int k, int lane, float* stage) {
    float mx = -INFINITY, pv[SLOTS];
    const int cnt = (n - lane + 31) >> 5;   // experts lane, lane + 32, ... below n
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        pv[j] = j < cnt ? l[lane + 32 * j] : -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        mx = fmaxf(mx, pv[j]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        pv[j] = j < cnt ? (float)exp((double)(pv[j] - mx)) : 0.f;
    }
    // sum in index order, the same on every lane: element e = 32*j + src comes from lane src, slot j
    float sum = 0.f;
    if (stage != nullptr) {
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            if (j < cnt) {
                stage[lane + 32 * j] = pv[j];
            }
        }
        __syncwarp();
        if (lane == 0) {
            if ((n & 3) == 0) {                 // rows of n floats: 16-byte aligned.  Loads ahead of the adds: one by one a token took 1.2 us longer
#pragma unroll 8
                for (int e = 0; e < n; e += 4) {
                    const float4 q = *reinterpret_cast<const float4*>(stage + e);
                    sum = (((sum + q.x) + q.y) + q.z) + q.w;
                }
            } else {
                for (int e = 0; e < n; ++e) {
                    sum += stage[e];
                }
            }
        }
        sum = __shfl_sync(0xffffffffu, sum, 0);
        __syncwarp();   // the row may be reused for the warp's next token
    } else {
        const int slots = (n + 31) >> 5;
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            if (j < slots) {
                const float mine_j = pv[j];
                const int live = min(32, n - 32 * j);
                for (int src = 0; src < live; ++src) {
                    sum += __shfl_sync(0xffffffffu, mine_j, src);
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < SLOTS; ++j) {
        pv[j] = pv[j] / sum;
    }
    unsigned used = 0u;
    float wsum = 0.f;
    float mine = 0.f;  // lane r keeps the r-th picked p and its expert
    int mine_e = 0;
    for (int r = 0; r < k; ++r) {
        unsigned best = 0u;   // bit pattern of the lane's largest remaining p (p >= 0: patterns order like values)
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            if (j < cnt && !(used & (1u << j))) {
                best = max(best, __float_as_uint(pv[j]));
            }
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best);
        unsigned cand = 0xffffffffu;   // lowest index on this lane that holds `top`
#pragma unroll
        for (int j = SLOTS - 1; j >= 0; --j) {
            if (j < cnt && !(used & (1u << j)) && __float_as_uint(pv[j]) == top) {
                cand = (unsigned)(lane + 32 * j);
            }
        }
        const int bi = (int)__reduce_min_sync(0xffffffffu, cand);
        if ((bi & 31) == lane) {
            used |= 1u << (bi >> 5);
        }
        const float bv = __uint_as_float(top);
        if (lane == (r & 31)) {
            mine = bv;
            mine_e = bi;
        }
        wsum += bv;
    }
    if (lane < k) {
        wt[lane] = mine / wsum;
        idx[lane] = mine_e;
    }
    return mine_e;
}

__device__ __forceinline__ int topk_of_token(const float* l, int* idx, float* wt,
                                             int n, int k, int lane, float* stage = nullptr) {
    if (n <= 128) {
        return topk_of_token_n<4>(l, idx, wt, n, k, lane, stage);
    } else if (n <= 256) {
        return topk_of_token_n<8>(l, idx, wt, n, k, lane, stage);
    }
    return topk_of_token_n<32>(l, idx, wt, n, k, lane, stage);
}

}  // namespace w4
