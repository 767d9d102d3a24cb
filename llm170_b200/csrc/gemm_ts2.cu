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
//   warp 0       tokens: this CTA's half, both k-blocks of a 128-channel stage as one TMA box per MMA, counted on CTA 0's barrier
//   warp 1       CTA 0: 8 x tcgen05.mma (M256, N tokens, K16) per stage; commits hand the stages back in both CTAs
//   warps 2-17   raw -> registers -> TMEM, four teams that take stages in turn; they arrive on the same barrier as the tokens
//   warp 18      weights and scales: raw int4 of the CTA's rows
//   warps 19-26  epilogue: accumulators -> shared memory -> TMA stores while the others are in the next tile
// Persistent: the roles run on from tile to tile, only the MMAs wait until the accumulators are read.  Tiles of up to 128 tokens alternate
// between two accumulators; larger ones take both.
//
// Grouped form (MoE prefill): token tiles from a device table, one expert's weights per tile; the epilogue rounds to f16 in shared memory,
// gives the accumulator back and applies SiLU(gate) * up there, or the routing weight on the way.
//
// What bounds it: the MMAs from 128 tokens on (256 x 7168 x 5120, tiles of 128: 18.6 us; 17.1 with the stores to TMEM taken out); on full waves
// the power limit, which holds the clock at about 1.35 GHz (4096 x 34816 x 5120: 1.56 PFLOP/s in bursts, 1.38 sustained, what a library f16
// GEMM does); below 128 tokens the expansion.  What it took, us per launch (start of each / with it):
//   scales with the weights, by TMA, and not through registers: 256 x 7168 x 5120, groups of 32: 25.2 / 19.8
//   one barrier per stage for tokens and weights, MMAs under a predicate, ring sizes known at compile time: 19.8 / 18.8 (an MMA costs its
//     issuer 50 cycles, a wait 100: with 128 tokens 8 MMAs of 64 cycles hardly cover them; two MMAs of half the tokens do where they are full)
//   teams instead of 16 warps on every stage: MoE layer of 128 experts, top-8, 2048 x 768, 256 tokens: 139 / 120, 4096 tokens: 375 / 358
//   TMA stores instead of 16 bytes per thread: second matmul of that layer, 4096 tokens: 139 / 107
// Tried and dropped: sigmoid by the hardware's power of two and reciprocal (no change); token boxes prefetched into L2 (no change); an output
// stage of 32 KB for 256 tokens, so that a fourth stage of tokens fits (the accumulators come back too late: 3000 tokens 262 / 284);
// two MMAs for tiles of up to 224 rows (3000 tokens 262 / 273).
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

constexpr int P_TEAM = 4, P_EXP_WARPS = 4 * P_TEAM;                  // expanding warps: teams that take stages in turn
constexpr int P_EPI_WARPS = 8;
constexpr int P_EPI0 = 3 + P_EXP_WARPS;                              // first warp of the epilogue
constexpr int P_THREADS = (3 + P_EXP_WARPS + P_EPI_WARPS) * 32;
constexpr int P_ROWS = 2 * TS_MROWS;                                 // weight rows of a pair's tile
constexpr int P_TOK_MAX = 256;
// Few tiles leave pairs idle: two to four pairs of a cluster share a tile's K, and their f32 sums meet in distributed shared memory, over the idle rings.
// us, weight rows with their clusters of single CTAs / so: 100 x 5120 x 17408 25.9 / 24.8, 128 x 5120 x 6144 17.1 / 14.2, 128 x 2560 x 9728 17.6 / 13.8,
// 128 x 3584 x 18944 in groups of 32 30.1 / 22.1.
constexpr int P_MAX_SPLIT = 4;
constexpr int P_SUB_MAX = P_TOK_MAX / 2;                             // tokens of an accumulator: a tile takes one or two
constexpr int P_RAW_STAGE = RAW_BYTES + ts_scale_bytes(32);          // raw weights and their scales, 128 channels
constexpr int P_OUT_STAGE = P_SUB_MAX * TS_MROWS * 2;                // f16 results of an accumulator on their way out, two of them
// Shared memory for tiles of at most `cap` tokens.  A team of expanding warps keeps to its stage of tokens and expanded weights, and to its
// raw stages (their number is a multiple of the teams'): it waits for every phase of the barriers that it looks at, so that the parity of
// a phase says which one it is.
__host__ __device__ constexpr int p_stages(int cap) { return cap <= 192 ? 4 : 3; }
__host__ __device__ constexpr int p_raw_stages(int cap) { return cap <= 128 ? 8 : cap <= 192 ? 4 : 6; }
__host__ __device__ constexpr int p_x_stage(int cap) { return cap / 2 * SK * 2; }                       // half of a tile's tokens
__host__ __device__ constexpr int p_off_x(int cap) { return p_raw_stages(cap) * P_RAW_STAGE; }
__host__ __device__ constexpr int p_off_out(int cap) { return p_off_x(cap) + p_stages(cap) * p_x_stage(cap); }
__host__ __device__ constexpr int p_off_bars(int cap) { return p_off_out(cap) + 2 * P_OUT_STAGE; }
__host__ __device__ constexpr int p_smem(int cap) { return p_off_bars(cap) + (2 * p_raw_stages(cap) + 2 * p_stages(cap) + 4) * 8 + 1024; }
constexpr int P_OUT_HALF = P_OUT_STAGE / 2;                          // 64 rows of all tokens: 128 bytes a token, 128B swizzle
constexpr int P_OUT_BOX = 32;                                        // tokens of a store
constexpr int P_X_BOXES = P_TOK_MAX / 32;                            // grouped form: token boxes of 16, 32, .. 128 rows, half of a tile
constexpr int P_TMEM_COLS = 512;                                     // 256 accumulator columns, four stages of 64
constexpr int P_GROUP_M = 8;                                         // token tiles that take turns on the same weights
static_assert(128 * TS_MROWS * 4 <= p_off_bars(128) && 192 * TS_MROWS * 4 <= p_off_bars(192) && 256 * TS_MROWS * 4 <= p_off_bars(256), "sums of a split");
static_assert(P_TOK_MAX + 4 * A_COLS <= P_TMEM_COLS, "TMEM");
static_assert(p_smem(128) <= 226 * 1024 && p_smem(192) <= 226 * 1024 && p_smem(256) <= 226 * 1024, "shared memory");

struct PairArgs {
    const uint32_t* qt;
    const uint32_t* st;
    void* out;
    int m, n, k;
    int out_f16;
    int m_tiles, n_tiles;
    int tok;                     // tokens per tile = MMA N (multiple of 32); grouped form: the most that a tile holds
    int ks;                      // K splits of a tile: that many pairs in a cluster, one tile each (dense)
    int halves;                  // 1: the second half of a tile's stages goes to an accumulator of its own (one tile of at most 128 tokens per pair)
    int split;                   // 1: a tile of more than 128 tokens is two MMAs (the grouped form's always are)
    int nrb_w;                   // 16-row blocks of the resident matrix (tile pitch)
    int pdl;
    float out_mul;
    uint32_t fma_add, fma_mul;   // as in gemm_ts.cu
    int* status;
    // grouped (MoE) form, as in gemm_ts.cu: token tiles of at most 256 rows from a device table, n = rows per expert
    const int* tile_expert;
    const int* tile_row0;
    const int* tile_rows;
    const int* num_tiles;
    int expert0;
    const float* row_w;
    int glu;
    int tables_fresh;
};
// Token boxes: of 16 (i + 1) rows (grouped form), or of a tile's MMAs; scales of a CTA's row blocks, 128 channels.
template <bool GROUPED>
struct PairMaps {
    CUtensorMap x[GROUPED ? P_X_BOXES : 2];
    CUtensorMap scales;
    CUtensorMap out[GROUPED ? 2 : 1];            // f16 results: 64 rows of 32 (grouped form: and of 8) tokens
};

// Issued by one lane of a warp that stays converged: under a predicate, not in a branch.
__device__ __forceinline__ void umma2_ts_f16(bool leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accum), "r"((uint32_t)leader)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair (`both`: a bit each, by rank in the cluster)
__device__ __forceinline__ void umma2_commit(bool leader, uint32_t bar, unsigned short both) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar),
        "h"(both), "r"((uint32_t)leader)
        : "memory");
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
// v += 16 columns of another accumulator
__device__ __forceinline__ void add_tmem16(uint32_t (&v)[16], uint32_t taddr) {
    uint32_t w[16];
    tmem_ld16(taddr, w);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        v[q] = __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(w[q]));
    }
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&h)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3])
                 : "memory");
}

// CAP: the most tokens of a tile.  (Ring sizes known at compile time: the MMAs' addresses cost their issuer fewer instructions, 256 x 7168 x
// 5120, tiles of 128, 19.5 -> 17.9 us.)
template <int GROUP, bool FMA, bool GROUPED, int CAP, bool SPLIT, bool HALVES>
__device__ __forceinline__ void pair_gemm(const PairMaps<GROUPED>& maps, const PairArgs& a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ __half2 s_row_w[GROUPED ? P_TOK_MAX / 2 : 1];         // routing weights of both accumulators' tokens
    if (GROUPED && a.tables_fresh) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    constexpr int GPS = SK / GROUP;                                  // scale groups per stage: 1 or 4
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1;                            // in the pair; CTA 0 issues the MMAs
    const int ks = SPLIT ? a.ks : 1, ksplit = SPLIT ? (int)(blockIdx.x >> 1) % ks : 0;
    const unsigned short both = (unsigned short)(3u << (2 * ksplit));
    auto in_leader = [&](uint32_t addr) {
        uint32_t r;
        if (SPLIT) {
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(2 * ksplit));
        } else {
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
        }
        return r;
    };
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;     // the same offset in both CTAs
    unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
    constexpr int X_STAGE = p_x_stage(CAP), NS = p_stages(CAP), NR = p_raw_stages(CAP);
    static_assert(X_STAGE % 1024 == 0 && p_off_x(CAP) % 1024 == 0 && p_off_out(CAP) % 1024 == 0 && NR % NS == 0, "operand alignment, phases");
    auto raw_addr = [&](int s) { return base + (uint32_t)s * P_RAW_STAGE; };
    auto x_addr = [&](int s) { return base + (uint32_t)(p_off_x(CAP) + s * X_STAGE); };
    const uint32_t bars = base + (uint32_t)p_off_bars(CAP);
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_free = [&](int s) { return bars + 8u * (NR + s); };
    auto full = [&](int s) { return bars + 8u * (2 * NR + s); };                // of CTA 0: both CTAs' tokens and expanded weights
    auto free_ = [&](int s) { return bars + 8u * (2 * NR + NS + s); };
    auto accum_bar = [&](int s) { return bars + 8u * (2 * NR + 2 * NS + s); };
    auto acc_free = [&](int s) { return bars + 8u * (2 * NR + 2 * NS + 2 + s); };     // of CTA 0

    // this pair's stages, of the tile's or of its part of K; the last of all may hold one k-block (32-channel groups)
    const int nst_all = (a.k / BK + 1) / 2, st0 = nst_all * ksplit / ks, nst = nst_all * (ksplit + 1) / ks - st0, nkb = min(a.k / BK - 2 * st0, 2 * nst);
    const int tiles = (GROUPED ? *a.num_tiles : a.m_tiles) * a.n_tiles;
    const int pair0 = (int)(blockIdx.x >> 1) / ks, pairs = (int)(gridDim.x >> 1) / ks;
    const bool halves = HALVES && a.halves != 0 && nst > 1;
    // Dense: groups of P_GROUP_M token tiles, whose neighbours share the weights: a wave's weights and tokens both stay within the L2.
    // Grouped: neighbours share the token rows, then the expert's weights; the table goes by size, the largest tiles first.
    struct Tile {
        int m0, rows, tok;                                           // tok: with padding, a multiple of 32
        int n0, rb0, nrbv;
    };
    auto expert_of = [&](int i) { return GROUPED && i < tiles ? a.tile_expert[i / a.n_tiles] - a.expert0 : 0; };
    auto place = [&](int i, int& mt, int& nt) {
        if (GROUPED) {
            mt = i / a.n_tiles;
            nt = i - mt * a.n_tiles;
        } else {
            const int g = i / (P_GROUP_M * a.n_tiles), m_first = g * P_GROUP_M;
            const int gm = min(P_GROUP_M, a.m_tiles - m_first), r = i - g * (P_GROUP_M * a.n_tiles);
            nt = r / gm;
            mt = m_first + r - nt * gm;
        }
    };
    auto tokens_at = [&](int i, Tile& t) {
        int mt, nt;
        place(i, mt, nt);
        t.m0 = GROUPED ? a.tile_row0[mt] : mt * a.tok;
        t.rows = GROUPED ? a.tile_rows[mt] : min(a.tok, a.m - t.m0);
        t.tok = GROUPED ? (t.rows + 31) & ~31 : a.tok;
        t.n0 = nt * P_ROWS + rank * TS_MROWS;
    };
    auto weights_at = [&](int i, int expert, Tile& t) {
        int mt, nt;
        place(i, mt, nt);
        t.n0 = nt * P_ROWS + rank * TS_MROWS;
        // rows that CTA 1 has nothing of: it expands CTA 0's once more, and stores nothing
        const int nl = t.n0 < a.n ? t.n0 : t.n0 - TS_MROWS;
        t.rb0 = (expert * a.n + nl) / TILE_ROWS;
        t.nrbv = min(TS_MROWS, a.n - nl) / TILE_ROWS;
    };
    // A tile of more than 128 tokens takes both accumulators: in two MMAs of half its tokens each (multiples of 32), or in one.  Of each
    // MMA's tokens a CTA holds half, both k-blocks of a stage behind one another.
    auto split = [&](int tok) { return tok > P_SUB_MAX && (GROUPED ? tok > 224 : a.split != 0); };
    auto first_mma = [&](int tok) { return split(tok) ? (tok / 2 + 31) & ~31 : tok; };

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < NR; ++s) {
            mbar_init(raw_full(s), 1);
            mbar_init(raw_free(s), P_TEAM);
        }
        for (int s = 0; s < NS; ++s) {
            mbar_init(full(s), 1 + 2 * P_TEAM);
            mbar_init(free_(s), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(accum_bar(s), 1);
            mbar_init(acc_free(s), 2 * P_EPI_WARPS);
        }
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
            Tile tl;
            tokens_at(i, tl);
            const int n0 = first_mma(tl.tok), n1 = tl.tok - n0;
            const CUtensorMap *map0 = &maps.x[GROUPED ? n0 / 32 - 1 : 0], *map1 = &maps.x[GROUPED && n1 > 0 ? n1 / 32 - 1 : 1];
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)NS && !__all_sync(0xffffffffu, mbar_wait(free_(sx), px, abort_flag, a.status, (61 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    if (rank == 0) {
                        mbar_expect_tx(full(sx), (uint32_t)(tl.tok * (SK * 2)));     // both CTAs' tokens (zeros past the end)
                    }
                    tma2_load_3d(x_addr(sx), map0, 0, tl.m0 + rank * (n0 / 2), 2 * (st0 + it), in_leader(full(sx)));
                    if (n1 > 0) {
                        tma2_load_3d(x_addr(sx) + (uint32_t)(n0 * SK), map1, 0, tl.m0 + n0 + rank * (n1 / 2), 2 * (st0 + it), in_leader(full(sx)));
                    }
                }
                __syncwarp();
                if (++sx == NS) {
                    sx = 0;
                    px ^= 1;
                }
            }
        }
        // CTA 0's commits arrive here too: all of them, before this CTA leaves
        for (int q = 0; q < NS && ok; ++q) {
            ok = __all_sync(0xffffffffu, mbar_wait(free_(sx), px, abort_flag, a.status, (69 << 16)));
            if (++sx == NS) {
                sx = 0;
                px ^= 1;
            }
        }
    } else if (warp == 2 + P_EXP_WARPS) {
        // ------------------------------------------------------------------ weights (they do not depend on the previous kernel)
        const bool leader = elect_one();
        int sr = 0;
        uint32_t pr = 1, cnt = 0;
        for (int i = pair0; i < tiles && ok; i += pairs) {
            Tile tl;
            weights_at(i, expert_of(i), tl);
            const uint32_t kb_bytes = (uint32_t)tl.nrbv * (TILE_WORDS * 4);
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)NR && !__all_sync(0xffffffffu, mbar_wait(raw_free(sr), pr, abort_flag, a.status, (62 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    const int kbs = min(2, nkb - 2 * it);
                    mbar_expect_tx(raw_full(sr), kbs * kb_bytes + ts_scale_bytes(GROUP));   // (scales past the end: zeros)
                    tma_load_2d(raw_addr(sr) + RAW_BYTES, &maps.scales, (st0 + it) * GPS * 8, tl.rb0, raw_full(sr));
                    const uint32_t* src = a.qt + ((size_t)(2 * (st0 + it)) * a.nrb_w + tl.rb0) * TILE_WORDS;
                    bulk_load(raw_addr(sr), src, kb_bytes, raw_full(sr));
                    if (kbs == 2) {
                        bulk_load(raw_addr(sr) + RAW_BYTES / 2, src + (size_t)a.nrb_w * TILE_WORDS, kb_bytes, raw_full(sr));
                    }
                }
                __syncwarp();
                if (++sr == NR) {
                    sr = 0;
                    pr ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();
        // Between two tiles the pipe would idle while an accumulator is read.  So the last two stages of a tile and the first two of the next
        // go through the first accumulator before the second: each is read while the other one is multiplied into.
        int sa = 0;
        uint32_t pa = 0, used = 0;                                   // used: accumulators so far
        auto tok_at = [&](int i) {
            Tile t;
            tokens_at(i, t);
            return t.tok;
        };
        auto in_time = [&](bool in) { return __all_sync(0xffffffffu, in) != 0; };
        auto acc_ready = [&](uint32_t u) {                           // read before it is written again
            return u < 2 || in_time(mbar_wait(acc_free(u & 1), ((u >> 1) - 1) & 1, abort_flag, a.status, (63 << 16)));
        };
        auto stage_ready = [&](int ba, uint32_t qa, int it) { return in_time(mbar_wait(full(ba), qa, abort_flag, a.status, (64 << 16) | it)); };
        // one stage into one accumulator: `n` of the tile's tokens, `off` bytes into the stage's tokens
        auto multiply = [&](int ba, int it, uint32_t acc, int n, uint32_t off, bool first) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(P_ROWS >> 4) << 24);
            const uint64_t db = umma_desc(x_addr(ba) + off);
            const uint64_t db1 = db + ((uint32_t)(n * BK) >> 4);
            const uint32_t ta = tmem_a + (uint32_t)(ba * A_COLS);
            const bool two = 2 * it + 1 < nkb;
#pragma unroll
            for (int j = 0; j < BK / 16; ++j) {
                umma2_ts_f16(leader, acc, ta + j * 8, db + 2 * j, idesc, (!first || j > 0) ? 1u : 0u);
            }
            if (two) {
#pragma unroll
                for (int j = 0; j < BK / 16; ++j) {
                    umma2_ts_f16(leader, acc, ta + BK / 2 + j * 8, db1 + 2 * j, idesc, 1u);
                }
            }
        };
        auto hand_back = [&]() {
            umma2_commit(leader, free_(sa), both);
            if (++sa == NS) {
                sa = 0;
                pa ^= 1;
            }
        };
        auto complete = [&](uint32_t u) { umma2_commit(leader, accum_bar(u & 1), both); };
        int tok_next = pair0 < tiles ? tok_at(pair0) : 0;
        for (int i = pair0; rank == 0 && i < tiles && ok; i += pairs) {
            const int tok = __shfl_sync(0xffffffffu, tok_next, 0);
            if (i + pairs < tiles) {
                tok_next = tok_at(i + pairs);
            }
            if (!split(tok)) {
                const bool two = tok > P_SUB_MAX;                    // (tiles that take both come first, so `used` is even here)
                const uint32_t acc = tmem + (used & 1) * P_SUB_MAX;
                const int half = (nst + 1) / 2;
                ok = acc_ready(used) && (!two || acc_ready(used + 1));
                for (int it = 0; it < nst && ok; ++it) {
                    ok = stage_ready(sa, pa, it);
                    if (ok) {
                        const int it0 = halves && it >= half ? half : 0;
                        multiply(sa, it, it0 > 0 ? acc + P_SUB_MAX : acc, tok, 0, it == it0);
                        hand_back();
                    }
                }
                complete(used++);
                if (two) {
                    complete(used++);
                }
                continue;
            }
            const uint32_t acc0 = tmem + (used & 1) * P_SUB_MAX, acc1 = tmem + (~used & 1) * P_SUB_MAX;
            const int n0 = first_mma(tok), n1 = tok - n0;
            const uint32_t off1 = (uint32_t)(n0 * SK);
            ok = acc_ready(used);
            for (int it = 0; it < nst && ok;) {
                const bool both = (it == 0 || it == nst - 2) && it + 1 < nst;
                const int ba = sa + 1 == NS ? 0 : sa + 1;
                const uint32_t qa = sa + 1 == NS ? pa ^ 1 : pa;
                const int next = both ? it + 2 : it + 1;
                ok = stage_ready(sa, pa, it);
                if (ok) {
                    multiply(sa, it, acc0, n0, 0, it == 0);
                    if (both) {
                        ok = stage_ready(ba, qa, it + 1);
                        if (ok) {
                            multiply(ba, it + 1, acc0, n0, 0, false);
                        }
                    }
                }
                if (next == nst) {
                    complete(used);
                }
                ok = ok && (it > 0 || acc_ready(used + 1));
                if (ok) {
                    multiply(sa, it, acc1, n1, off1, it == 0);
                    hand_back();
                    if (both) {
                        multiply(sa, it + 1, acc1, n1, off1, false);
                        hand_back();
                    }
                }
                it = next;
            }
            complete(used + 1);
            used += 2;
        }
    } else if (warp < 2 + P_EXP_WARPS) {
        // ------------------------------------------------------------------ expand: raw int4 -> f16 in TMEM
        // A team of four warps takes a stage, the teams take stages in turn (ts_expand_stage; with three stages the fourth team has nothing to do).
        const int quad = warp & 3, team = (warp - 2) >> 2;
        Tile tl{};
        int expert = pair0 < tiles ? expert_of(pair0) : 0;
        const uint32_t td = tmem_a + ((uint32_t)(quad * 32) << 16) + (uint32_t)(team * A_COLS);
        int sr = team, skip = team;                                  // skip: stages of the other teams before this one's next
        uint32_t pr = 0, pa = 1, cnt = 0;
        for (int i = pair0; team < NS && i < tiles && ok; i += pairs) {
            weights_at(i, expert, tl);
            expert = expert_of(i + pairs);
            int it = skip;
            for (; it < nst && ok; it += NS, ++cnt) {
                ok = ts_expand_stage<GROUP, FMA>(
                    raw_addr(sr), quad, tl.nrbv, lane, td, a.fma_add, a.fma_mul,
                    [&]() { return __all_sync(0xffffffffu, mbar_wait(raw_full(sr), pr, abort_flag, a.status, (66 << 16) | it)) != 0; },
                    [&]() { return cnt == 0 || __all_sync(0xffffffffu, mbar_wait(free_(team), pa, abort_flag, a.status, (67 << 16) | it)) != 0; },
                    [&]() { mbar_arrive(raw_free(sr)); }, [&]() { mbar_arrive_cluster(in_leader(full(team))); });
                pa ^= 1;
                if ((sr += NS) >= NR) {
                    sr = team;
                    pr ^= 1;
                }
            }
            skip = it - nst;
        }
    } else if (SPLIT) {
        // ------------------------------------------------------------------ this pair's sums, for the pairs of the cluster
        // [token][row] f32 over the rings, which are idle: every MMA is complete
        const int quad = warp & 3, sub = (warp - P_EPI0) >> 2;
        Tile tl;
        tokens_at(pair0, tl);
        ok = mbar_wait(accum_bar(0), 0, abort_flag, a.status, (68 << 16)) && (tl.tok <= P_SUB_MAX || mbar_wait(accum_bar(1), 0, abort_flag, a.status, (68 << 16)));
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int c0 = sub * 16; ok && c0 < tl.rows; c0 += P_EPI_WARPS / 4 * 16) {
            uint32_t v[16];
            tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
            if (halves) {
                add_tmem16(v, tmem + P_SUB_MAX + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0);
            }
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                *reinterpret_cast<float*>(base_ptr + ((c0 + q) * TS_MROWS + quad * 32 + lane) * 4) = __uint_as_float(v[q]);
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int quad = warp & 3, sub = (warp - P_EPI0) >> 2;
        const int lrow = quad * 32 + lane, et = (int)threadIdx.x - P_EPI0 * 32;
        const bool glu = GROUPED && a.glu != 0, weighted = GROUPED && a.row_w != nullptr;
        unsigned char* stage_ptr = base_ptr + p_off_out(CAP);
        const uint32_t stage = base + (uint32_t)p_off_out(CAP);
        // stmatrix: lane (j, r) addresses token r of the 8 x 8 block j & 1 (rows) of token octet j >> 1
        const int st_chunk = ((quad & 1) * 4 + sub * 2 + ((lane >> 3) & 1)) ^ (lane & 7);
        const uint32_t st_base = (uint32_t)((quad >> 1) * P_OUT_HALF + (((lane >> 4) << 3) + (lane & 7)) * 128 + st_chunk * 16);
        const uint32_t t_ld = tmem + ((uint32_t)(quad * 32 + sub * 16) << 16);
        uint32_t used = 0;
        for (int i = pair0; i < tiles; i += pairs) {
            Tile tl;
            tokens_at(i, tl);
            const int rows_out = max(0, min(TS_MROWS, a.n - tl.n0));
            const int n0 = split(tl.tok) ? first_mma(tl.tok) : min(tl.tok, P_SUB_MAX);
            const bool f16 = GROUPED || a.out_f16;
            if (f16) {
                if (et == 0) {                                       // the stage's last stores have read it: all, or all but the other accumulator's
                    if (n0 < tl.tok) {
                        bulk_wait_group_read<0>();
                    } else {
                        bulk_wait_group_read<1>();
                    }
                }
                if (weighted && et < tl.rows) {
                    const uint32_t b = et < n0 ? used & 1 : ~used & 1;
                    reinterpret_cast<__half*>(s_row_w)[b * P_SUB_MAX + (et < n0 ? et : et - n0)] = __float2half_rn(a.row_w[tl.m0 + et]);
                }
                asm volatile("bar.sync 1, %0;" ::"n"(P_EPI_WARPS * 32) : "memory");
            }
            const uint32_t used0 = used;
            for (int t0 = 0; t0 < tl.tok; t0 += n0, ++used) {
                const int n = min(n0, tl.tok - t0), rows = min(n, tl.rows - t0);         // tokens of this accumulator, without padding
                const uint32_t b = used & 1, acc = b * P_SUB_MAX;
                ok = ok && mbar_wait(accum_bar(used & 1), (used >> 1) & 1, abort_flag, a.status, (68 << 16));
                ok = __all_sync(0xffffffffu, ok);
                if (a.pdl && used == 0) {
                    asm volatile("griddepcontrol.wait;" ::: "memory");   // outputs may be what the previous kernel still reads
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (ok && f16) {
                    // Through shared memory and TMA stores of 64 rows by 32 tokens: 16 rows x 32 tokens from TMEM in the fragment layout
                    // that stmatrix transposes, into the 128B swizzle of the stores (no bank conflicts).
                    for (int c0 = 0; c0 < rows; c0 += 64) {
                        uint32_t v[32];
                        tmem_ld_16x256b_x4(t_ld + acc + (uint32_t)c0, v);
                        if (c0 + 32 < n) {
                            tmem_ld_16x256b_x4(t_ld + acc + (uint32_t)c0 + 32u, v + 16);
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (halves) {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                if (c0 + 32 * hh < n) {
                                    uint32_t w[16];
                                    tmem_ld_16x256b_x4(t_ld + P_SUB_MAX + (uint32_t)(c0 + 32 * hh), w);
                                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                                    for (int q = 0; q < 16; ++q) {
                                        v[16 * hh + q] = __float_as_uint(__uint_as_float(v[16 * hh + q]) + __uint_as_float(w[q]));
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            uint32_t h[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                __half2 p = __floats2half2_rn(__uint_as_float(v[8 * q + 2 * j]) * a.out_mul, __uint_as_float(v[8 * q + 2 * j + 1]) * a.out_mul);
                                if (weighted) {                      // as mul_row_w: the f16 sum times the f16 weight
                                    p = __hmul2(p, s_row_w[b * (P_SUB_MAX / 2) + ((c0 + q * 16 + (j >> 1) * 8) >> 1) % (P_SUB_MAX / 2) + (lane & 3)]);
                                }
                                h[j] = *reinterpret_cast<const uint32_t*>(&p);
                            }
                            if (c0 + q * 16 < n) {
                                stmatrix_x4_trans(stage + b * P_OUT_STAGE + st_base + (uint32_t)((c0 + q * 16) * 128), h);
                            }
                        }
                    }
                } else if (ok) {
                    for (int c0 = sub * 16; c0 < rows; c0 += P_EPI_WARPS / 4 * 16) {
                        uint32_t v[16];
                        tmem_ld16(tmem + acc + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
                        if (halves) {
                            add_tmem16(v, tmem + P_SUB_MAX + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0);
                        }
#pragma unroll
                        for (int q = 0; q < 16; ++q) {
                            if (c0 + q < rows && lrow < rows_out) {
                                reinterpret_cast<float*>(a.out)[(size_t)(tl.m0 + t0 + c0 + q) * a.n + tl.n0 + lrow] = __uint_as_float(v[q]) * a.out_mul;
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(in_leader(acc_free(used & 1)));
                }
            }
            if (!f16) {
                continue;
            }
            if (glu) {
                // The activation comes here, where the next tile's MMAs run beside it.  Of 32 rows the first 16 are gate sums, the others
                // the up sums of the same outputs.  A warp takes four tokens at a time and writes their 64 outputs over the first half of
                // what it read.
                asm volatile("bar.sync 1, %0;" ::"n"(P_EPI_WARPS * 32) : "memory");
                const int c = lane & 7, gate = (c >> 2) * P_OUT_HALF, gc = ((c >> 1) & 1) * 4 + (c & 1);
                for (int r0 = (warp - P_EPI0) * 4; ok && r0 < tl.rows; r0 += P_EPI_WARPS * 4) {
                    const bool second = r0 >= n0;                    // (n0 is a multiple of 32)
                    const int tok = r0 - (second ? n0 : 0) + (lane >> 3);
                    unsigned char* row = stage_ptr + ((used0 + second) & 1) * P_OUT_STAGE + tok * 128;
                    uint4 v = *reinterpret_cast<const uint4*>(row + gate + (gc ^ (tok & 7)) * 16);
                    const uint4 up = *reinterpret_cast<const uint4*>(row + gate + ((gc + 2) ^ (tok & 7)) * 16);
                    __half2* h = reinterpret_cast<__half2*>(&v);
                    const __half2* hu = reinterpret_cast<const __half2*>(&up);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 g2 = __half22float2(h[q]), u2 = __half22float2(hu[q]);
                        h[q] = __halves2half2(silu_mul_f16(g2.x, u2.x), silu_mul_f16(g2.y, u2.y));
                    }
                    __syncwarp();
                    *reinterpret_cast<uint4*>(row + (c ^ (tok & 7)) * 16) = v;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync 1, %0;" ::"n"(P_EPI_WARPS * 32) : "memory");
            const int col = glu ? tl.n0 / 2 : tl.n0, boxes = rows_out == 0 ? 0 : glu || rows_out <= TS_MROWS / 2 ? 1 : 2;
            for (int t0 = 0, u = (int)used0; t0 < tl.tok; t0 += n0, ++u) {
                const int rows = min(min(n0, tl.tok - t0), tl.rows - t0), m0 = tl.m0 + t0;
                const int whole = GROUPED ? rows & ~(P_OUT_BOX - 1) : rows;           // dense: what lies past the last token is not written
                if (et == 0) {
                    for (int hf = 0; hf < boxes && ok; ++hf) {
                        const uint32_t src = stage + (uint32_t)((u & 1) * P_OUT_STAGE + hf * P_OUT_HALF);
                        for (int r = 0; r < whole; r += P_OUT_BOX) {
                            tma_store_2d(&maps.out[0], src + (uint32_t)(r * 128), col + hf * 64, m0 + r);
                        }
                        if (GROUPED) {
                            for (int r = whole; r + 8 <= rows; r += 8) {
                                tma_store_2d(&maps.out[GROUPED ? 1 : 0], src + (uint32_t)(r * 128), col + hf * 64, m0 + r);
                            }
                        }
                    }
                    bulk_commit_group();
                }
                if (GROUPED && ok) {                                 // the last tokens of an expert, next to another one's
                    const int n_out = glu ? a.n / 2 : a.n, r = (rows & ~7) + (et >> 4), c = et & 15;
                    if (r < rows && c < rows_out / (glu ? 16 : 8)) {
                        *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(a.out) + (size_t)(m0 + r) * n_out + col + c * 8) =
                            *reinterpret_cast<const uint4*>(stage_ptr + (u & 1) * P_OUT_STAGE + (c >> 3) * P_OUT_HALF + r * 128 + ((c & 7) ^ (r & 7)) * 16);
                    }
                }
            }
        }
    }
    if (SPLIT) {
        // Every CTA adds an equal share of its rows' results over all splits, in their order.
        __syncthreads();
        cluster_sync_all();
        if (a.pdl) {
            asm volatile("griddepcontrol.wait;" ::: "memory");           // outputs may be what the previous kernel still reads
        }
        Tile tl;
        tokens_at(pair0, tl);
        const int nr4 = max(0, min(TS_MROWS, a.n - tl.n0)) / 4, total = tl.rows * nr4;
        const int e0 = total * ksplit / ks, e1 = total * (ksplit + 1) / ks;
        for (int e = e0 + (int)threadIdx.x; e < e1 && !*abort_flag; e += P_THREADS) {
            const int tok = e / nr4, r = (e - tok * nr4) * 4;
            float4 pv[P_MAX_SPLIT];
#pragma unroll
            for (int s = 0; s < P_MAX_SPLIT; ++s) {
                pv[s] = s < ks ? ld_dsmem_f32x4(base + (uint32_t)((tok * TS_MROWS + r) * 4), (unsigned)(2 * s + rank)) : make_float4(0, 0, 0, 0);
            }
            float4 sum = pv[0];
#pragma unroll
            for (int s = 1; s < P_MAX_SPLIT; ++s) {
                if (s < ks) {
                    sum.x += pv[s].x;
                    sum.y += pv[s].y;
                    sum.z += pv[s].z;
                    sum.w += pv[s].w;
                }
            }
            const size_t o = (size_t)(tl.m0 + tok) * a.n + tl.n0 + r;
            if (a.out_f16) {
                const __half2 h0 = __floats2half2_rn(sum.x * a.out_mul, sum.y * a.out_mul), h1 = __floats2half2_rn(sum.z * a.out_mul, sum.w * a.out_mul);
                *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(a.out) + o) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
            } else {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + o) =
                    make_float4(sum.x * a.out_mul, sum.y * a.out_mul, sum.z * a.out_mul, sum.w * a.out_mul);
            }
        }
    }
    if (warp == P_EPI0 && lane == 0) {
        bulk_wait_group_read<0>();                                   // the last stores have read this CTA's shared memory
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();                                              // nothing of the other CTA still reads or signals this one
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P_TMEM_COLS) : "memory");
    }
}

template <int GROUP, bool FMA, bool GROUPED, int CAP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_ts2_kernel(const __grid_constant__ PairMaps<GROUPED> maps, const PairArgs a) {
    pair_gemm<GROUP, FMA, GROUPED, CAP, false, false>(maps, a);
}
// Sums in two halves (one tile of at most 128 tokens per pair).
template <int GROUP, bool FMA>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1) gemm_ts2_halves_kernel(const __grid_constant__ PairMaps<false> maps, const PairArgs a) {
    pair_gemm<GROUP, FMA, false, P_SUB_MAX, false, true>(maps, a);
}
// (a kernel of its own: a launch that names the size of its clusters, and K ranges known only then, cost 0.6 us)
template <int GROUP, bool FMA, int CAP>
__global__ void __launch_bounds__(P_THREADS, 1) gemm_ts2_split_kernel(const __grid_constant__ PairMaps<false> maps, const PairArgs a) {
    pair_gemm<GROUP, FMA, false, CAP, true, (CAP <= P_SUB_MAX)>(maps, a);
}

}  // namespace

namespace {
template <int GROUP, bool FMA>
auto pair_split_kernel(int tok) {
    return tok <= 128 ? gemm_ts2_split_kernel<GROUP, FMA, 128> : tok <= 192 ? gemm_ts2_split_kernel<GROUP, FMA, 192> : gemm_ts2_split_kernel<GROUP, FMA, 256>;
}
template <int GROUP, bool FMA, bool GROUPED>
auto pair_kernel(int tok) {
    return tok <= 128 ? gemm_ts2_kernel<GROUP, FMA, GROUPED, 128> : tok <= 192 ? gemm_ts2_kernel<GROUP, FMA, GROUPED, 192> : gemm_ts2_kernel<GROUP, FMA, GROUPED, 256>;
}
}  // namespace

cudaError_t gemm_ts2_init_device() {
    cudaError_t e = cudaSuccess;
    for (int tok : {128, 192, 256}) {
        for (const void* f : {(const void*)pair_kernel<128, false, false>(tok), (const void*)pair_kernel<128, true, false>(tok), (const void*)pair_kernel<32, false, false>(tok),
                              (const void*)pair_kernel<128, false, true>(tok), (const void*)pair_kernel<128, true, true>(tok), (const void*)pair_kernel<32, false, true>(tok),
                              (const void*)pair_split_kernel<128, false>(tok), (const void*)pair_split_kernel<128, true>(tok), (const void*)pair_split_kernel<32, false>(tok)}) {
            if (e == cudaSuccess) {
                e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, p_smem(tok));
            }
        }
    }
    for (const void* f : {(const void*)gemm_ts2_halves_kernel<128, false>, (const void*)gemm_ts2_halves_kernel<128, true>, (const void*)gemm_ts2_halves_kernel<32, false>}) {
        if (e == cudaSuccess) {
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, p_smem(P_SUB_MAX));
        }
    }
    return e;
}

// Tokens per tile with the least estimated time (microseconds, fitted to 1238 measurements on B200 within a third of their shape's best: 22 shapes
// of 1792..34816 rows, K 1536..17408, 14 batches of 72..3000 tokens, seven tile widths; good to 4.2 %): 3.14 and 0.0064 per token of the tile per
// launch; a stage of 128 channels takes 0.009 + 0.00212 per token, the rate of the MMAs, but not less than the expansion (0.193 us, groups of
// 32: 0.221), and with all pairs busy, when power holds the clock down, 0.05 + 0.00272 per token and at least 0.268 (0.326); each further tile
// of a pair 0.48 where tiles take both accumulators.  f32 results, stored from registers, take another 0.0263 per token less 3.23 with each tile
// (202 measurements before the accumulators alternated).
// K splits (up to `max_split`, where all clusters are resident at once): the stages of a tile are dealt to two to four pairs of a cluster, which takes
// another 0.01 us per token for the sums and, with all pairs busy, 2.73 us and 0.067 per stage (330 measurements, 15 shapes of 1024..34816 rows,
// 12..250 tokens; good to 3.6 %).  `min_parts`: in place of weight rows that split K in so many parts -- no accumulator takes more stages than there.
TsChoice Dec::gemm_ts2_choose(const Lin* l, int t, int out_kind, int max_split, int min_parts) const {
    TsChoice best{0, 0, 1e30};
    const int n_tiles = (l->n + P_ROWS - 1) / P_ROWS, stages = (l->k + SK - 1) / SK, pairs = sm_count / 2;
    const bool g128 = l->group == 128;
    for (int cap = P_TOK_MAX; cap >= 64; cap -= 32) {
        const int m_tiles = (t + cap - 1) / cap;
        const int tok = ((t + m_tiles - 1) / m_tiles + 31) / 32 * 32;
        const long long tiles = (long long)m_tiles * n_tiles, waves = (tiles + pairs - 1) / pairs;
        const double full = std::min(1.0, std::max(0.0, ((double)tiles / (waves * pairs) - 0.46) / 0.54));
        const double light = std::max(g128 ? 0.193 : 0.221, 0.009 + 0.00212 * tok);
        const double heavy = std::max(g128 ? 0.268 : 0.326, 0.05 + 0.00272 * tok);
        const double f32 = out_kind == W4A16_OUT_F16 ? 0.0 : std::max(0.0, 0.0263 * tok - 3.23);
        const double c = 3.14 + 0.0064 * tok + waves * (stages * (light + std::max(0.0, heavy - light) * full) + f32) + (waves - 1) * (tok > P_SUB_MAX ? 0.48 : 0.0);
        const int halves = tok <= P_SUB_MAX ? 2 : 1;                 // (as in gemm_ts2)
        if (c < best.cost && (min_parts <= 1 || (min_parts <= halves && tiles <= pairs))) {
            best = TsChoice{tok, 1, c};
        }
        for (int ks = 2; ks <= max_split && ks <= stages && tiles <= ts_clusters[1][2 * ks]; ++ks) {
            const double busy = std::min(1.0, std::max(0.0, ((double)tiles * ks / pairs - 0.46) / 0.54));
            const int nst = (stages + ks - 1) / ks;
            const double cs = 3.14 + 0.0164 * tok + nst * (light + std::max(0.0, heavy - light) * busy) + (double)tiles * ks / pairs * (2.73 + 0.067 * nst);
            if (cs < best.cost && min_parts <= ks * halves) {
                best = TsChoice{tok, ks, cs};
            }
        }
    }
    return best;
}

namespace {
// One tensor map over f16 [rows][k]: boxes of `box_rows` rows by both k-blocks of a stage.
CUresult pair_map(EncodeTiledFn enc, CUtensorMap* map, const void* x, int rows, int k, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)BK, (cuuint64_t)rows, (cuuint64_t)(k / BK)};
    const cuuint64_t strides[2] = {(cuuint64_t)k * 2, (cuuint64_t)BK * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// f16 results [rows][n]: boxes of 64 columns by `box_rows` rows, 128B swizzle.
CUresult pair_out_map(EncodeTiledFn enc, CUtensorMap* map, void* out, int rows, int n, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)n * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, out, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

template <bool GROUPED>
cudaError_t launch_pairs(const Lin* l, const PairMaps<GROUPED>& maps, PairArgs& a, int tiles, int sm_count, cudaStream_t st) {
    a.qt = l->qt;
    a.st = (const uint32_t*)l->st;
    a.k = l->k;
    a.nrb_w = l->n / TILE_ROWS;
    a.out_mul = l->out_mul;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * (a.ks > 1 ? tiles * a.ks : std::min(tiles, sm_count / 2)));
    cfg.blockDim = dim3(P_THREADS);
    cfg.dynamicSmemBytes = a.tok <= 128 ? p_smem(128) : a.tok <= 192 ? p_smem(192) : p_smem(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (a.pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (!GROUPED && a.ks > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 2 * a.ks;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    const bool fma = l->group == 128 && l->fma_e >= 0;
    if (fma) {
        const __half2 mul = __float2half2_rn(ldexpf(-8.0f, -l->fma_e));
        memcpy(&a.fma_mul, &mul, sizeof(mul));
        a.fma_add = ((uint32_t)(20 - l->fma_e) << 26) + ((uint32_t)(24 - l->fma_e) << 10);
        a.out_mul = ldexpf(l->out_mul, l->fma_e);
    }
    if constexpr (!GROUPED) {
        if (a.ks == 1 && a.halves) {
            return cudaLaunchKernelEx(&cfg, l->group != 128 ? gemm_ts2_halves_kernel<32, false> : fma ? gemm_ts2_halves_kernel<128, true> : gemm_ts2_halves_kernel<128, false>, maps, a);
        }
        if (a.ks > 1) {
            return cudaLaunchKernelEx(&cfg, l->group != 128 ? pair_split_kernel<32, false>(a.tok) : fma ? pair_split_kernel<128, true>(a.tok) : pair_split_kernel<128, false>(a.tok), maps, a);
        }
    }
    return cudaLaunchKernelEx(&cfg, l->group != 128 ? pair_kernel<32, false, GROUPED>(a.tok) : fma ? pair_kernel<128, true, GROUPED>(a.tok) : pair_kernel<128, false, GROUPED>(a.tok), maps, a);
}
}  // namespace

// `short_sums`: in place of weight rows that would split K.  An MMA's sum drops what lies below the accumulator's last bit, so the error of a result grows
// with the stages that go through one accumulator (6144 channels in three parts 2.4e-6 of the results' size, in one 7.2e-6).  A pair with one tile of
// at most 128 tokens has a second accumulator to spare: half of its stages go there, and both are added at the end.
int Dec::gemm_ts2(const Lin* l, const void* x, void* dst, int t, int out_kind, int tok, int ks, bool short_sums, cudaStream_t st) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    PairMaps<false> maps;
    CUresult cr = ts_scale_map(enc, &maps.scales, l->st, l->n, l->k, l->group);
    // Two MMAs keep the pipe busy from tile to tile, at 8 cycles more than one each below 128 tokens: 512 x 5120 x 17408, tiles of 192, one
    // MMA / two 71.5 / 74.8 us, 1024 x 5120 x 17408, tiles of 160, 131 / 147; full ones cost nothing.
    const int split = ks == 1 && tok > 192, n0 = split ? (tok / 2 + 31) & ~31 : tok;             // as in the kernel
    for (int i = 0; i < 2 && cr == CUDA_SUCCESS; ++i) {
        cr = pair_map(enc, &maps.x[i], x, t, l->k, (i == 1 && split ? tok - n0 : n0) / 2);
    }
    if (cr == CUDA_SUCCESS) {
        cr = pair_out_map(enc, &maps.out[0], dst, t, l->n, P_OUT_BOX);   // (f32 results are stored from registers)
    }
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    PairArgs a{};
    a.tok = tok;
    a.ks = ks;
    a.m_tiles = (t + tok - 1) / tok;
    a.n_tiles = (l->n + P_ROWS - 1) / P_ROWS;
    a.out = dst;
    a.m = t;
    a.n = l->n;
    a.out_f16 = out_kind == W4A16_OUT_F16;
    a.split = split;
    a.halves = short_sums && tok <= P_SUB_MAX && (ks > 1 || a.m_tiles * a.n_tiles <= sm_count / 2);
    a.pdl = tune_pdl ? 1 : 0;
    a.status = gemm_status;
    const cudaError_t e = launch_pairs<false>(l, maps, a, a.m_tiles * a.n_tiles, sm_count, st);
    if (e != cudaSuccess) {
        return cuda_fail("launch gemm", e);
    }
    last_kernel = "gemm_ts2_kernel<" + std::to_string(l->group) + (l->fma_e >= 0 ? ",fma> " : "> ") + std::to_string(tok) + "-token tiles" + (ks > 1 ? ", ksplit " + std::to_string(ks) : "") +
                  (a.halves ? ", sums in halves" : "");
    launches++;
    return 0;
}

// Grouped form over expert segments, as Dec::gemm_ts_grouped; the table's tiles hold at most `bm` rows (128, 192 or 256), the largest
// come first.
int Dec::gemm_ts2_grouped(const Lin* l, const void* xs, int xs_rows, void* out, int n_per_expert, const MoeBufs& b, int max_tiles,
                          int bm, const float* row_w, cudaStream_t st, bool tables_fresh) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    PairMaps<true> maps;
    CUresult cr = ts_scale_map(enc, &maps.scales, l->st, l->n, l->k, l->group);
    for (int i = 0; i < P_X_BOXES && cr == CUDA_SUCCESS; ++i) {
        cr = pair_map(enc, &maps.x[i], xs, xs_rows, l->k, 16 * (i + 1));
    }
    for (int i = 0; i < 2 && cr == CUDA_SUCCESS; ++i) {
        cr = pair_out_map(enc, &maps.out[i], out, xs_rows, l->glu_f > 0 ? n_per_expert / 2 : n_per_expert, i == 0 ? P_OUT_BOX : 8);
    }
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    PairArgs a{};
    a.tok = bm;
    a.ks = 1;
    a.n_tiles = (n_per_expert + P_ROWS - 1) / P_ROWS;
    a.out = out;
    a.m = xs_rows;
    a.n = n_per_expert;
    a.out_f16 = 1;
    a.pdl = tune_pdl ? 1 : 0;
    a.status = gemm_status;
    a.tile_expert = b.tile_expert;
    a.tile_row0 = b.tile_row0;
    a.tile_rows = b.tile_rows;
    a.num_tiles = b.n_tiles;
    a.expert0 = moe.e0;
    a.row_w = row_w;
    a.glu = l->glu_f > 0 ? 1 : 0;
    a.tables_fresh = tables_fresh ? 1 : 0;
    const cudaError_t e = launch_pairs<true>(l, maps, a, max_tiles * a.n_tiles, sm_count, st);
    if (e != cudaSuccess) {
        return cuda_fail("launch grouped gemm", e);
    }
    last_kernel = "gemm_ts2_kernel<" + std::to_string(l->group) + (l->fma_e >= 0 ? ",fma" : "") + ",grouped>";
    launches++;
    return 0;
}

}  // namespace w4
