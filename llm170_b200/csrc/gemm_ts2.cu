// W4A16 prefill GEMM on CTA pairs:  y[m][n] = sum_k x[m][k] * f16((q[n][k]-8)*s[n][k/g]).
//
// Takes the place of the reference's prefill GEMMs (crates/backend-gpu/src/rawcuda/w4a16_dec/kernels/marlin.rs:94-213) for
// large batches.  Like them it multiplies the dequantised weight ROUNDED ONCE TO F16 and accumulates in f32.
//
// Two CTAs on neighbouring SMs compute a tile of 256 weight rows x up to 256 tokens with tcgen05.mma.cta_group::2: each holds its 128
// weight rows as the A operand in its TMEM (expanded there straight from registers, as in gemm_ts.cu) and half of the tokens as the B
// operand in its shared memory.  Per k-block of 64 an SM then reads 16 KB of operands from shared memory and writes 20 KB in the 512 cycles
// of its MMAs; the 256 x 256 tiles of gemm_tc.cu read 96 KB, write 72 KB in 1024, more than the 128 bytes a cycle that there are.
//
//   warp 0       tokens: this CTA's half, both k-blocks of a 128-channel stage as one TMA box, counted on CTA 0's barrier
//   warp 1       CTA 0: 8 x tcgen05.mma (M256, N tokens, K16) per stage; commits hand the stages back in both CTAs
//   warps 2-9    raw -> registers -> TMEM, one 16-row block each; they arrive on CTA 0's barrier
//   warp 10      weights: raw int4 of the CTA's rows
//   warps 11-18  epilogue: accumulators -> shared memory -> global while the others are in the next tile
// Persistent: the roles run on from tile to tile, only the MMAs wait until the accumulators are read.
//
// What bounds it: the MMAs at 192 tokens and more (the expansion and its TMEM stores taken out: 5 % less time at 512 x 5120 x 6144,
// 256 tokens; half of the MMAs taken out: 29 % less), the expansion at 128 and below; on full waves the power limit, which holds the clock at
// about 1.35 GHz (4096 x 34816 x 5120: 1.38 PFLOP/s, what a library f16 GEMM sustains).  About 5 us of a launch and 2 us of a tile are entry,
// first loads and epilogue.  4096 tokens, one layer of 7168 x 5120, 5120 x 6144, 34816 x 5120, 5120 x 17408: 2310 -> 2090 us against the
// token-row form, 1024 tokens 629 -> 565.  The epilogue with two-byte stores and half the stage: 12 % more at 512 x 34816 x 5120 (143.6
// against 123.1 us).
// Every wait is bounded: on expiry the kernel records a status code and all roles fall through to the common exit.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/w4a16_b200.h"
#include "dec.h"
#include "gemm_ts.cuh"

namespace w4 {

namespace {

constexpr int P_EPI_WARPS = 8;
constexpr int P_EPI0 = 3 + DQ_WARPS;                                 // first warp of the epilogue
constexpr int P_THREADS = (3 + DQ_WARPS + P_EPI_WARPS) * 32;
constexpr int P_ROWS = 2 * TS_MROWS;                                 // weight rows of a pair's tile
constexpr int P_NX = 4, P_NR = 4, P_NA = 4;                          // token, raw weight and expanded weight stages of 128 channels
constexpr int P_TOK_MAX = 256;
constexpr int P_X_STAGE = P_TOK_MAX / 2 * SK * 2;                    // 32 KB: half of the tile's tokens
constexpr int P_OUT_STAGE = P_TOK_MAX * TS_MROWS * 2;                // f16 results on their way out: [token][row]
constexpr int P_OFF_X = P_NR * RAW_BYTES, P_OFF_OUT = P_OFF_X + P_NX * P_X_STAGE, P_OFF_BARS = P_OFF_OUT + P_OUT_STAGE;
constexpr int P_BARS = 2 * P_NR + 2 * P_NX + 2 * P_NA + 2;
constexpr int P_SMEM = P_OFF_BARS + P_BARS * 8 + 1024;
constexpr int P_TMEM_COLS = 512;                                     // 256 accumulator columns, four stages of 64
constexpr int P_GROUP_M = 8;                                         // token tiles that take turns on the same weights
static_assert(P_TOK_MAX + P_NA * A_COLS <= P_TMEM_COLS, "TMEM");
static_assert(P_SMEM <= 226 * 1024, "shared memory");

struct PairArgs {
    const uint32_t* qt;
    const uint32_t* st;
    void* out;
    int m, n, k;
    int out_f16;
    int m_tiles, n_tiles;
    int tok;                     // tokens per tile = MMA N (multiple of 32)
    int nrb_w;                   // 16-row blocks of the resident matrix (tile pitch)
    int pdl;
    float out_mul;
    uint32_t fma_add, fma_mul;   // as in gemm_ts.cu
    int* status;
};

__device__ __forceinline__ void umma2_ts_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accum)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma2_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((unsigned short)3)
                 : "memory");
}
__device__ __forceinline__ uint32_t in_leader(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// What the barriers order across the pair is TMEM (tcgen05.wait and the tcgen05 fences) and TMA writes (complete_tx), no memory that
// a thread reads or writes: release at cluster scope, which waits for all of a thread's stores, took 0.9 us per stage.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// TMA load into this CTA's shared memory, counted on a barrier of the pair's first CTA
__device__ __forceinline__ void tma2_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
// 16 TMEM lanes x 32 columns, registers as in tmem_st_16x256b_x4; the caller waits
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&h)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                 : "memory");
}

template <int GROUP, bool FMA>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_ts2_kernel(const __grid_constant__ CUtensorMap tmap_x, const PairArgs a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    constexpr int GPS = SK / GROUP;                                  // scale groups per stage: 1 or 4
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1;                            // in the pair; CTA 0 issues the MMAs
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;     // the same offset in both CTAs
    unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
    const uint32_t x_half = (uint32_t)a.tok * BK;                    // bytes of one k-block of this CTA's tokens: tok / 2 rows
    auto raw_addr = [&](int s) { return base + (uint32_t)s * RAW_BYTES; };
    auto x_addr = [&](int s) { return base + (uint32_t)(P_OFF_X + s * P_X_STAGE); };
    const uint32_t bars = base + (uint32_t)P_OFF_BARS;
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_free = [&](int s) { return bars + 8u * (P_NR + s); };
    auto x_full = [&](int s) { return bars + 8u * (2 * P_NR + s); };                          // of CTA 0: both halves
    auto x_free = [&](int s) { return bars + 8u * (2 * P_NR + P_NX + s); };
    auto a_ready = [&](int s) { return bars + 8u * (2 * P_NR + 2 * P_NX + s); };              // of CTA 0: both CTAs' rows
    auto a_free = [&](int s) { return bars + 8u * (2 * P_NR + 2 * P_NX + P_NA + s); };
    const uint32_t accum_bar = bars + 8u * (2 * P_NR + 2 * P_NX + 2 * P_NA), acc_free = accum_bar + 8u;   // the latter of CTA 0

    const int nkb = a.k / BK, nst = (nkb + 1) / 2;                   // the last stage may hold one k-block (32-channel groups)
    const int tiles = a.m_tiles * a.n_tiles;
    const int pair0 = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    // Groups of P_GROUP_M token tiles, whose neighbours share the weights: a wave's weights and tokens both stay within the L2.
    struct Tile {
        int m0, rows, n0, rb0, nrbv;
    };
    auto tile_at = [&](int i) {
        const int g = i / (P_GROUP_M * a.n_tiles), m_first = g * P_GROUP_M;
        const int gm = min(P_GROUP_M, a.m_tiles - m_first), r = i - g * (P_GROUP_M * a.n_tiles);
        const int nt = r / gm;
        Tile t;
        t.m0 = (m_first + r - nt * gm) * a.tok;
        t.rows = min(a.tok, a.m - t.m0);
        t.n0 = nt * P_ROWS + rank * TS_MROWS;
        // rows that CTA 1 has nothing of: it expands CTA 0's once more, and stores nothing
        const int nl = t.n0 < a.n ? t.n0 : t.n0 - TS_MROWS;
        t.rb0 = nl / TILE_ROWS;
        t.nrbv = min(TS_MROWS, a.n - nl) / TILE_ROWS;
        return t;
    };

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < P_NR; ++s) {
            mbar_init(raw_full(s), 1);
            mbar_init(raw_free(s), DQ_WARPS);
        }
        for (int s = 0; s < P_NX; ++s) {
            mbar_init(x_full(s), 1);
            mbar_init(x_free(s), 1);
        }
        for (int s = 0; s < P_NA; ++s) {
            mbar_init(a_ready(s), 2 * DQ_WARPS);
            mbar_init(a_free(s), 1);
        }
        mbar_init(accum_bar, 1);
        mbar_init(acc_free, 2 * P_EPI_WARPS);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(P_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                                              // both CTAs' barriers and TMEM are there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (a.pdl) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    const uint32_t tmem_a = tmem + (uint32_t)P_TOK_MAX;              // A ring: [stage][64 columns]
    volatile int* abort_flag = &s_abort;

    // After a wait that ran out a role leaves its loops; the epilogue goes on through its own without waiting or loading, so that its
    // named barrier stays matched.
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------------ tokens: this CTA's half of the tile
        if (a.pdl) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }
        const bool leader = elect_one();
        int sx = 0;
        uint32_t px = 1, cnt = 0;
        for (int i = pair0; i < tiles && ok; i += pairs) {
            const Tile tl = tile_at(i);
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)P_NX && !__all_sync(0xffffffffu, mbar_wait(x_free(sx), px, abort_flag, a.status, (61 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    if (rank == 0) {
                        mbar_expect_tx(x_full(sx), 4 * x_half);      // both k-blocks (zeros past the end) of both halves
                    }
                    tma2_load_3d(x_addr(sx), &tmap_x, 0, tl.m0 + rank * (a.tok / 2), 2 * it, in_leader(x_full(sx)));
                }
                __syncwarp();
                if (++sx == P_NX) {
                    sx = 0;
                    px ^= 1;
                }
            }
        }
        // CTA 0's commits arrive here too: all of them, before this CTA leaves
        for (int q = 0; q < P_NX && ok; ++q) {
            ok = __all_sync(0xffffffffu, mbar_wait(x_free(sx), px, abort_flag, a.status, (69 << 16)));
            if (++sx == P_NX) {
                sx = 0;
                px ^= 1;
            }
        }
    } else if (warp == 2 + DQ_WARPS) {
        // ------------------------------------------------------------------ weights (they do not depend on the previous kernel)
        const bool leader = elect_one();
        int sr = 0;
        uint32_t pr = 1, cnt = 0;
        for (int i = pair0; i < tiles && ok; i += pairs) {
            const Tile tl = tile_at(i);
            const uint32_t kb_bytes = (uint32_t)tl.nrbv * (TILE_WORDS * 4);
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)P_NR && !__all_sync(0xffffffffu, mbar_wait(raw_free(sr), pr, abort_flag, a.status, (62 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    const int kbs = min(2, nkb - 2 * it);
                    mbar_expect_tx(raw_full(sr), kbs * kb_bytes);
                    const uint32_t* src = a.qt + ((size_t)(2 * it) * a.nrb_w + tl.rb0) * TILE_WORDS;
                    bulk_load(raw_addr(sr), src, kb_bytes, raw_full(sr));
                    if (kbs == 2) {
                        bulk_load(raw_addr(sr) + RAW_BYTES / 2, src + (size_t)a.nrb_w * TILE_WORDS, kb_bytes, raw_full(sr));
                    }
                }
                __syncwarp();
                if (++sr == P_NR) {
                    sr = 0;
                    pr ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(a.tok >> 3) << 17) | ((uint32_t)(P_ROWS >> 4) << 24);
        int sx = 0, sa = 0;
        uint32_t px = 0, pa = 0, done = 0;
        for (int i = pair0; rank == 0 && i < tiles && ok; i += pairs, ++done) {
            // the accumulators are read before they are written again
            if (done > 0 && !__all_sync(0xffffffffu, mbar_wait(acc_free, (done - 1) & 1, abort_flag, a.status, (63 << 16)))) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int it = 0; it < nst; ++it) {
                const bool in = mbar_wait(x_full(sx), px, abort_flag, a.status, (64 << 16) | it) &&
                                mbar_wait(a_ready(sa), pa, abort_flag, a.status, (65 << 16) | it);
                if (!__all_sync(0xffffffffu, in)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t db = umma_desc(x_addr(sx));
                const uint64_t db1 = db + (x_half >> 4);
                const uint32_t ta = tmem_a + (uint32_t)(sa * A_COLS);
                const bool two = 2 * it + 1 < nkb;
                if (leader) {
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j) {
                        umma2_ts_f16(tmem, ta + j * 8, db + 2 * j, idesc, (it > 0 || j > 0) ? 1u : 0u);
                    }
                    if (two) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) {
                            umma2_ts_f16(tmem, ta + BK / 2 + j * 8, db1 + 2 * j, idesc, 1u);
                        }
                    }
                    umma2_commit(a_free(sa));
                    umma2_commit(x_free(sx));
                    if (it + 1 == nst) {
                        umma2_commit(accum_bar);
                    }
                }
                __syncwarp();
                if (++sx == P_NX) {
                    sx = 0;
                    px ^= 1;
                }
                if (++sa == P_NA) {
                    sa = 0;
                    pa ^= 1;
                }
            }
        }
    } else if (warp < 2 + DQ_WARPS) {
        // ------------------------------------------------------------------ expand: raw int4 -> f16 in TMEM
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int rb = quad * 2 + half;                              // a warp may touch the TMEM lanes 32 * (warp % 4) .. +31
        const int ng = a.k / GROUP;
        constexpr int SCQ = 4;                                       // scale loads in flight, as in gemm_ts.cu
        const uint32_t* sp = nullptr;
        int sleft = 0;
        uint32_t scq[SCQ], scn[SCQ];                                 // of this tile, and the first ones of the next
        auto load_scales = [&]() {
            const uint32_t v = sleft > 0 ? __ldg(sp) : 0u;
            sp += 32;
            sleft -= 32;
            return v;
        };
        auto first_scales = [&](int i) {
            const Tile tl = tile_at(i);
            const uint32_t* p = a.st + (size_t)(tl.rb0 + (rb < tl.nrbv ? rb : 0)) * ng * 8 + lane;
#pragma unroll
            for (int q = 0; q < SCQ; ++q) {
                scn[q] = ng * 8 - lane > 32 * q ? __ldg(p + 32 * q) : 0u;
            }
        };
        if (pair0 < tiles) {
            first_scales(pair0);
        }
        uint32_t sc_cur = 0;
        const uint32_t t_st = tmem_a + ((uint32_t)(quad * 32 + half * 16) << 16);
        int sr = 0, sa = 0;
        uint32_t pr = 0, pa = 1, cnt = 0;
        for (int i = pair0; i < tiles && ok; i += pairs) {
            const Tile tl = tile_at(i);
            const int rbl = rb < tl.nrbv ? rb : 0;
            sp = a.st + (size_t)(tl.rb0 + rbl) * ng * 8 + lane + 32 * SCQ;
            sleft = ng * 8 - lane - 32 * SCQ;
#pragma unroll
            for (int q = 0; q < SCQ; ++q) {
                scq[q] = scn[q];
            }
            if (i + pairs < tiles) {
                first_scales(i + pairs);
            }
            const uint32_t r_ld = base + (uint32_t)rbl * (TILE_WORDS * 4) + (uint32_t)lane * 16u;
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (!__all_sync(0xffffffffu, mbar_wait(raw_full(sr), pr, abort_flag, a.status, (66 << 16) | it))) {
                    ok = false;
                    break;
                }
                const uint32_t ra = r_ld + (uint32_t)sr * RAW_BYTES;
                const uint4 raw0 = lds128(ra);
                const uint4 raw1 = lds128(ra + RAW_BYTES / 2);       // stale bytes when the stage holds one k-block
                if (((it * GPS) & 3) == 0) {
                    sc_cur = scq[0];
#pragma unroll
                    for (int q = 0; q + 1 < SCQ; ++q) {
                        scq[q] = scq[q + 1];
                    }
                    scq[SCQ - 1] = load_scales();
                }
                uint32_t sc[GPS];
#pragma unroll
                for (int q = 0; q < GPS; ++q) {
                    sc[q] = __shfl_sync(0xffffffffu, sc_cur, ((it * GPS + q) & 3) * 8 + (lane >> 2));
                }
                uint32_t v[16];
                const TsScale<FMA> sc0(sc[0], a.fma_add, a.fma_mul), sc1(sc[GPS > 1 ? 1 : 0], a.fma_add, a.fma_mul);
                ts_expand<FMA>(raw0, sc0, sc1, v);
                if (cnt >= (uint32_t)P_NA && !__all_sync(0xffffffffu, mbar_wait(a_free(sa), pa, abort_flag, a.status, (67 << 16) | it))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t td = t_st + (uint32_t)(sa * A_COLS);
                tmem_st_16x256b_x4(td, v);
                if (GPS > 1) {
                    ts_expand<FMA>(raw1, TsScale<FMA>(sc[GPS > 2 ? 2 : 0], a.fma_add, a.fma_mul),
                                   TsScale<FMA>(sc[GPS > 2 ? 3 : 0], a.fma_add, a.fma_mul), v);
                } else {
                    ts_expand<FMA>(raw1, sc0, sc1, v);
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(raw_free(sr));                       // both k-blocks are in registers
                }
                tmem_st_16x256b_x4(td + BK / 2, v);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(in_leader(a_ready(sa)));
                }
                if (++sr == P_NR) {
                    sr = 0;
                    pr ^= 1;
                }
                if (++sa == P_NA) {
                    sa = 0;
                    pa ^= 1;
                }
            }
        }
        for (int q = 0; q < P_NA && ok; ++q) {                       // as with the tokens
            ok = __all_sync(0xffffffffu, mbar_wait(a_free(sa), pa, abort_flag, a.status, (70 << 16)));
            if (++sa == P_NA) {
                sa = 0;
                pa ^= 1;
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3, sub = (warp - P_EPI0) >> 2;
        const int lrow = quad * 32 + lane, et = (int)threadIdx.x - P_EPI0 * 32;
        constexpr int PER_TOK = TS_MROWS * 2;
        unsigned char* stage_ptr = base_ptr + P_OFF_OUT;
        // stmatrix: lane (j, r) addresses token r of the 8 x 8 block j & 1 (rows) of token octet j >> 1
        const int st_chunk = (quad * 4 + sub * 2 + ((lane >> 3) & 1)) ^ (lane & 7);
        const uint32_t st_base = base + (uint32_t)P_OFF_OUT + (uint32_t)((((lane >> 4) << 3) + (lane & 7)) * PER_TOK + st_chunk * 16);
        const uint32_t t_ld = tmem + ((uint32_t)(quad * 32 + sub * 16) << 16);
        uint32_t done = 0;
        for (int i = pair0; i < tiles; i += pairs, ++done) {
            const Tile tl = tile_at(i);
            const int rows_out = max(0, min(TS_MROWS, a.n - tl.n0));
            ok = ok && mbar_wait(accum_bar, done & 1, abort_flag, a.status, (68 << 16));
            ok = __all_sync(0xffffffffu, ok);
            if (a.pdl && done == 0) {
                asm volatile("griddepcontrol.wait;" ::: "memory");   // outputs may be what the previous kernel still reads
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (a.out_f16) {
                // Through shared memory, whole 16-byte pieces of a token's row: 16 rows x 32 tokens from TMEM in the fragment layout that
                // stmatrix transposes; the 16-byte pieces of a token lie exclusive-or'ed with the token (no bank conflicts).
                if (ok) {
                    for (int c0 = 0; c0 < tl.rows; c0 += 64) {
                        uint32_t v[32];
                        tmem_ld_16x256b_x4(t_ld + (uint32_t)c0, v);
                        if (c0 + 32 < a.tok) {
                            tmem_ld_16x256b_x4(t_ld + (uint32_t)c0 + 32u, v + 16);
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t h[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const __half2 p = __floats2half2_rn(__uint_as_float(v[8 * q + 2 * j]) * a.out_mul, __uint_as_float(v[8 * q + 2 * j + 1]) * a.out_mul);
                                h[j] = *reinterpret_cast<const uint32_t*>(&p);
                            }
                            if (c0 + q * 16 < a.tok) {
                                stmatrix_x4_trans(st_base + (uint32_t)((c0 + q * 16) * PER_TOK), h);
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(in_leader(acc_free));
                }
                asm volatile("bar.sync 1, %0;" ::"n"(P_EPI_WARPS * 32) : "memory");
                if (ok) {
                    const int pieces = rows_out / 8;
                    __half* out = reinterpret_cast<__half*>(a.out) + (size_t)tl.m0 * a.n + tl.n0;
                    for (int e = et; e < tl.rows * pieces; e += P_EPI_WARPS * 32) {
                        const int tok = e / pieces, c = e - tok * pieces;
                        *reinterpret_cast<uint4*>(out + (size_t)tok * a.n + c * 8) =
                            *reinterpret_cast<const uint4*>(stage_ptr + tok * PER_TOK + (c ^ (tok & 7)) * 16);
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"n"(P_EPI_WARPS * 32) : "memory");         // the stage is free again
            } else {
                if (ok) {
                    for (int c0 = sub * 16; c0 < tl.rows; c0 += P_EPI_WARPS / 4 * 16) {
                        uint32_t v[16];
                        tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            if (c0 + q < tl.rows && lrow < rows_out) {
                                reinterpret_cast<float*>(a.out)[(size_t)(tl.m0 + c0 + q) * a.n + tl.n0 + lrow] = __uint_as_float(v[q]) * a.out_mul;
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(in_leader(acc_free));
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                                              // nothing of the other CTA still reads or signals this one
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P_TMEM_COLS) : "memory");
    }
}

}  // namespace

cudaError_t gemm_ts2_init_device() {
    cudaError_t e = cudaSuccess;
    for (const void* f : {(const void*)gemm_ts2_kernel<128, false>, (const void*)gemm_ts2_kernel<128, true>, (const void*)gemm_ts2_kernel<32, false>}) {
        if (e == cudaSuccess) {
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM);
        }
    }
    return e;
}

// Tokens per tile with the least estimated time (microseconds, fitted to 700 measurements on B200: 140 shapes of 66..4096 tokens, 1024..34816
// rows, K 512..17408, five tile widths each): 5.4 us per launch and 1.7 per further tile of a pair; a stage of 128 channels takes 0.00224 us per
// token of the tile, the rate of the MMAs, but not less than the expansion (0.317 us, groups of 32: 0.445), and with all pairs busy, when
// power holds the clock down, 0.082 + 0.00254 per token and at least 0.439 (0.470).  f32 results, stored from registers while the MMAs wait for
// the accumulators, take another 0.0263 per token less 3.23 with each tile (202 measurements: 0.84..1.09 of them, nine tenths 0.94..1.06).
TsChoice Dec::gemm_ts2_choose(const Lin* l, int t, int out_kind) const {
    TsChoice best{0, 1, 1e30};
    const int n_tiles = (l->n + P_ROWS - 1) / P_ROWS, stages = (l->k + SK - 1) / SK, pairs = sm_count / 2;
    for (int cap = P_TOK_MAX; cap >= 96; cap -= 32) {
        const int m_tiles = (t + cap - 1) / cap;
        const int tok = ((t + m_tiles - 1) / m_tiles + 31) / 32 * 32;
        const long long tiles = (long long)m_tiles * n_tiles, waves = (tiles + pairs - 1) / pairs;
        const double full = std::min(1.0, std::max(0.0, ((double)tiles / (waves * pairs) - 0.41) / 0.52));
        const double light = std::max(l->group == 128 ? 0.317 : 0.445, 0.00224 * tok);
        const double heavy = std::max(l->group == 128 ? 0.439 : 0.470, 0.082 + 0.00254 * tok);
        const double f32 = out_kind == W4A16_OUT_F16 ? 0.0 : 0.0263 * tok - 3.23;
        const double c = 5.4 + waves * (stages * (light + std::max(0.0, heavy - light) * full) + f32) + (waves - 1) * 1.7;
        if (c < best.cost) {
            best = TsChoice{tok, 1, c};
        }
    }
    return best;
}

int Dec::gemm_ts2(const Lin* l, const void* x, void* dst, int t, int out_kind, int tok, cudaStream_t st) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    PairArgs a{};
    a.tok = tok;
    a.m_tiles = (t + tok - 1) / tok;
    a.n_tiles = (l->n + P_ROWS - 1) / P_ROWS;
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)BK, (cuuint64_t)t, (cuuint64_t)(l->k / BK)};
    const cuuint64_t strides[2] = {(cuuint64_t)l->k * 2, (cuuint64_t)BK * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)tok / 2, 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    a.qt = l->qt;
    a.st = (const uint32_t*)l->st;
    a.out = dst;
    a.m = t;
    a.n = l->n;
    a.k = l->k;
    a.out_f16 = out_kind == W4A16_OUT_F16;
    a.nrb_w = l->n / TILE_ROWS;
    a.pdl = tune_pdl ? 1 : 0;
    a.out_mul = l->out_mul;
    a.status = gemm_status;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * std::min(a.m_tiles * a.n_tiles, sm_count / 2));
    cfg.blockDim = dim3(P_THREADS);
    cfg.dynamicSmemBytes = P_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (a.pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    cudaError_t e;
    if (l->group != 128) {
        e = cudaLaunchKernelEx(&cfg, gemm_ts2_kernel<32, false>, map, a);
    } else if (l->fma_e < 0) {
        e = cudaLaunchKernelEx(&cfg, gemm_ts2_kernel<128, false>, map, a);
    } else {
        const __half2 mul = __float2half2_rn(ldexpf(-8.0f, -l->fma_e));
        memcpy(&a.fma_mul, &mul, sizeof(mul));
        a.fma_add = ((uint32_t)(20 - l->fma_e) << 26) + ((uint32_t)(24 - l->fma_e) << 10);
        a.out_mul = ldexpf(l->out_mul, l->fma_e);
        e = cudaLaunchKernelEx(&cfg, gemm_ts2_kernel<128, true>, map, a);
    }
    if (e != cudaSuccess) {
        return cuda_fail("launch gemm", e);
    }
    last_kernel = "gemm_ts2_kernel<" + std::to_string(l->group) + (l->fma_e >= 0 ? ",fma> " : "> ") + std::to_string(tok) + "-token tiles";
    launches++;
    return 0;
}

}  // namespace w4
