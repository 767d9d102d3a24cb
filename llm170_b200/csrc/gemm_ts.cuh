// Pieces shared by the weight-row GEMM kernels (gemm_ts.cu, gemm_ts2.cu): weights expanded in registers and stored to TMEM.
#pragma once
#include <cstdint>

#include "gemm_common.cuh"
#include "gemv_common.cuh"
#include "ptx.cuh"

namespace w4 {

constexpr int TS_MROWS = 128;                   // weight rows per MMA
constexpr int BK = TILE_K;
constexpr int SK = 2 * BK;                      // channels per stage: two k-blocks, one 128-channel scale group
constexpr int RAW_BYTES = TS_MROWS * SK / 2;    // 8 KB per stage
constexpr int A_COLS = SK / 2;                  // TMEM columns of one expanded stage (two f16 per column)
constexpr int DQ_WARPS = TS_MROWS / TILE_ROWS;  // a warp per 16-row block
// Scales of a raw stage, behind its weights: [row block][group][8] words, one TMA box.  Read by the lanes from global memory instead, four
// loads ahead, they held up every stage: the wait for the stores to TMEM took those reads along.  us per launch before / now: 27 tokens of
// 34816 x 5120 29.2 / 27.2, of 5120 x 17408 19.7 / 18.7; groups of 32: 27 tokens 33.8 / 31.0, 197 tokens of 34816 x 5120 64.8 / 56.6.
__host__ __device__ constexpr int ts_scale_bytes(int group) { return DQ_WARPS * (SK / group) * 32; }

// Scale words [16-row blocks][groups][8] of a matrix: boxes of a stage's groups by the row blocks of a CTA.
inline CUresult ts_scale_map(EncodeTiledFn enc, CUtensorMap* map, void* st, int n, int k, int group) {
    const int ng = k / group;
    const cuuint64_t dims[2] = {(cuuint64_t)ng * 8, (cuuint64_t)(n / TILE_ROWS)};
    const cuuint64_t strides[1] = {(cuuint64_t)ng * 32};
    const cuuint32_t box[2] = {(cuuint32_t)(SK / group * 8), (cuuint32_t)DQ_WARPS};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, st, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// 16 TMEM lanes x 32 columns from one warp: register 4i + {0,1} of lane (g, t) -> row g, columns 8i + 2t + {0,1};
// register 4i + {2,3} -> row g + 8
__device__ __forceinline__ void tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_dsmem_f32x4(uint32_t local_addr, unsigned cta_rank) {
    uint32_t ra;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local_addr), "r"(cta_rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
    return v;
}
// Scale pair (rows g, g + 8) of a tile's 32 or more channels, ready for ts_expand: f16((q - 8) * s) as (q - 8) times s, or (FMA) as a
// multiply-add of the raw nibble with s scaled by powers of two and -8 s 2^-E (Dec::fma_shift).
template <bool FMA>
struct TsScale {
    uint32_t s0, s1, c0, c1;
    __device__ __forceinline__ TsScale(uint32_t s2, uint32_t add, uint32_t mul) {
        const uint32_t sp = FMA ? s2 + add : s2;           // exponents up by 24 - E (rows g) and 20 - E (rows g + 8): no field overflows
        s0 = __byte_perm(sp, sp, 0x1010);
        s1 = __byte_perm(sp, sp, 0x3232);
        if (FMA) {
            const uint32_t c = hmul2u(s2, mul);
            c0 = __byte_perm(c, c, 0x1010);
            c1 = __byte_perm(c, c, 0x3232);
        }
    }
};
// A lane's 16 raw bytes of a tile -> its 16 registers of tcgen05.st.16x256b.x4: sa / sb = scales of the first / second 32 channels.
template <bool FMA>
__device__ __forceinline__ void ts_expand(const uint4& raw, const TsScale<FMA>& sa, const TsScale<FMA>& sb, uint32_t (&v)[16]) {
    const uint32_t rw[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const TsScale<FMA>& s = w < 2 ? sa : sb;
        uint32_t f[4];
        if (FMA) {
            nibbles_as_subnormals(rw[w], f);
            v[4 * w + 0] = hfma2u(f[0], s.s0, s.c0);
            v[4 * w + 1] = hfma2u(f[2], s.s0, s.c0);
            v[4 * w + 2] = hfma2u(f[1], s.s1, s.c1);
            v[4 * w + 3] = hfma2u(f[3], s.s1, s.c1);
        } else {
            dequant_word(rw[w], f);
            v[4 * w + 0] = hmul2u(f[0], s.s0);
            v[4 * w + 1] = hmul2u(f[2], s.s0);
            v[4 * w + 2] = hmul2u(f[1], s.s1);
            v[4 * w + 3] = hmul2u(f[3], s.s1);
        }
    }
}

// One warp's part of a stage: the two 16-row blocks of the TMEM lanes that it may touch (32 * (warp % 4) .. +31), expanded from the raw stage at
// `raw` into the stage at `td`.  A stage's way -- wait, expand, wait, store, hand over -- is a chain of about 600 cycles: teams of four warps
// take stages in turn, so that the chains of several stages overlap, where eight warps with a row block each went through every stage
// together.  A team keeps to its slots of the rings (their numbers are multiples of the teams'): it waits for every phase of the barriers that
// it looks at, so the parity of a phase says which one it is.
template <int GROUP, bool FMA, class Full, class Free, class RawRead, class Ready>
__device__ __forceinline__ bool ts_expand_stage(uint32_t raw, int quad, int nrbv, int lane, uint32_t td, uint32_t fma_add, uint32_t fma_mul,
                                                Full&& wait_full, Free&& wait_free, RawRead&& raw_read, Ready&& ready) {
    constexpr int GPS = SK / GROUP;                                  // scale groups per stage: 1 or 4
    if (!wait_full()) {
        return false;
    }
    constexpr int SPK = GPS > 1 ? 2 : 1;                             // scale groups per k-block
    const int rb[2] = {quad * 2 < nrbv ? quad * 2 : 0, quad * 2 + 1 < nrbv ? quad * 2 + 1 : 0};
    uint4 w[2][2];                                                   // [k-block][row block] (stale bytes when there is no second k-block)
    uint32_t sc[2][2][SPK];                                          // scale pairs of the lane's rows
    auto load = [&](int kb) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            w[kb][b] = lds128(raw + (uint32_t)(kb * (RAW_BYTES / 2) + rb[b] * (TILE_WORDS * 4)) + (uint32_t)lane * 16u);
#pragma unroll
            for (int q = 0; q < SPK; ++q) {
                sc[kb][b][q] = lds32(raw + RAW_BYTES + (uint32_t)(rb[b] * (GPS * 32) + (GPS > 1 ? kb * 64 : 0) + q * 32) + (uint32_t)(lane >> 2) * 4u);
            }
        }
    };
    load(0);
    if (!wait_free()) {
        return false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int b = q & 1, kb = q >> 1;
        const TsScale<FMA> s0(sc[kb][b][0], fma_add, fma_mul);
        uint32_t v[16];
        if (GPS > 1) {
            ts_expand<FMA>(w[kb][b], s0, TsScale<FMA>(sc[kb][b][SPK - 1], fma_add, fma_mul), v);
        } else {
            ts_expand<FMA>(w[kb][b], s0, s0, v);
        }
        if (q == 0) {
            load(1);
        }
        tmem_st_16x256b_x4(td + ((uint32_t)(b * 16) << 16) + (uint32_t)(kb * (BK / 2)), v);
    }
    // The stage goes back when the last of what was read of it has been used: an arrival before that could pass loads under way, and the copy
    // into the stage is not ordered behind them.
    __syncwarp();
    if (lane == 0) {
        raw_read();
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        ready();
    }
    return true;
}

}  // namespace w4
