// W4A16 GEMM with the weights as the TMEM operand:  y[m][n] = sum_k x[m][k] * f16((q[n][k]-8)*s[n][k/g]).
//
// Takes the place of the reference's small-batch FFMA family and of its prefill GEMMs
// (crates/backend-gpu/src/rawcuda/assets/gptq4.cu:44-723, kernels/marlin.rs:94-213) above the decode path's eight rows.
// Like them it multiplies the dequantised weight ROUNDED ONCE TO F16 and accumulates in f32.
//
// The 128 rows of an MMA are WEIGHT rows and its N columns are tokens, so a batch of 9 tokens multiplies a 16-wide tile,
// not a padded 128-row one.  The expanded weights never touch shared memory: a warp reads a raw int4 tile, expands it in
// registers and stores it to TMEM (tcgen05.st.16x256b: the T64 layout keeps a lane's nibbles in exactly that register
// order), where tcgen05.mma reads it as its A operand; the tokens are the shared-memory operand.
//
//   warp 0      tokens: both k-blocks of a 128-channel stage as one TMA box (128B swizzle, shallow ring: L2)
//   warp 1      issues 8 x tcgen05.mma (M128, N tokens, K16) per stage; commits hand the TMEM stage and the token stage back
//   warps 2-    raw -> registers -> TMEM, then the epilogue (the first eight): three teams of four warps that take stages in turn, or
//               eight warps with a 16-row block of every stage each
//   last warp   weights: raw int4 of the CTA's rows (one bulk copy per k-block) and their scales, deep ring: this hides the HBM latency
//
// What bounds it: below about 64 tokens neither HBM nor the tensor pipe but the serial chain of a role per stage (wait,
// issue, hand over; 34816 x 5120, 16 tokens, two CTAs per SM: 0.69 us per stage of 2 x 8 KB).  So the roles that issue
// TMA, bulk copies and MMAs each have a warp of their own that stays converged with one elected lane (uniform registers
// feed these instructions: 36 -> 34 us) and a stage is one token box and two weight copies (34 -> 30.6 us).  The expansion
// itself, the TMEM stores, loads from HBM and the MMAs each cost under 15 % when taken out alone; what is left is the chain of the
// expanding warps, about 600 cycles a stage, so up to 64 tokens (96 where CTAs queue) teams of four take stages in turn, and three chains
// overlap: 27 tokens of 34816 x 5120 27.2 -> 25.6 us, of 5120 x 17408 18.7 -> 18.4, in groups of 32 31.0 -> 28.9.  Above that the MMAs
// of a stage take as long as its chain, with fewer than four stages per CTA a team is idle: eight warps on every stage.
// 256 rows per CTA were slower (33.5 us).  With teams a stage takes 550 cycles, the stages of two CTAs on an SM 430 each, 230 of them the MMAs: each of its 32 KB is
// written to TMEM and read from it once, and the two do not overlap (34816 x 5120, 27 tokens: 22.8 us; with stages handed over in halves 39).
//
// The K splits of a tile form a thread-block cluster and sum their f32 accumulators through distributed shared memory in
// split order (no global scratch, no tickets).
// Launched with programmatic stream serialization: raw weights are requested before the dependency wait.
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

constexpr int TS_TEAM = 4, TS_MAX_TEAMS = 3;    // expanding warps: teams that take stages in turn, or a warp per 16-row block on every stage
__host__ __device__ constexpr int ts_threads(bool teams) { return (3 + (teams ? TS_MAX_TEAMS * TS_TEAM : DQ_WARPS)) * 32; }
constexpr int TSG_THREADS = ts_threads(false);  // grouped form (teams: 2 to 6 % slower, 60 and fewer rows per expert)
constexpr int TS_XBOX = 64;                     // grouped form: rows of a token box
constexpr int TS_STAGE_BYTES = 16 * 1024;       // grouped form: results on their way out
constexpr int RED_TOK = 64;                     // tokens per round of the cluster's sum
__host__ __device__ constexpr int ts_push_pitch(int tok) { return tok + 4; }   // floats of a row on their way to its owner: conflict-free 16-byte accesses
// K splits whose sums are sent to their owners instead of being read there.  Sending costs a 16-byte piece per lane where reading has rows of 128 bytes, and room
// beside the rings.  Sent against read, us at 16 / 32 / 48 / 64 tokens: 7168 x 5120 in clusters of 4 8.4 / 9.1 / 10.5 / 11.8 against 8.7 / 9.4 / 10.2 / 11.1;
// 5120 x 17408 in clusters of 6 15.2 / 15.7 / 18.3 / 19.8 against 15.7 / 16.4 / 17.0 / 18.4; 2560 x 2560 in clusters of 7 4.8 / 5.5 / 6.8 / 8.0 against
// 4.8 / 5.2 / 5.8 / 6.6; 4096 x 4096, 32-channel groups, in clusters of 4 5.9 / 6.6 / 7.2 / 7.9 against 6.3 / 7.1 / 7.4 / 7.9.
constexpr bool ts_pushes(int tok, int ks) { return ks > 1 && tok <= 32 && tok * ks <= 192; }
// Shared memory requested per CTA.  The lower bounds keep CTAs whose TMEM does not fit together off one SM: a CTA that
// waits for TMEM columns would hold up its cluster, and the columns may belong to a CTA that waits for its own cluster.
// Half the TMEM: two CTAs per SM, never three; all of it: alone, also beside a CTA of the other kind.
constexpr size_t TS_SMEM_HALF_MIN = 77 * 1024, TS_SMEM_HALF_MAX = 112 * 1024;
constexpr size_t TS_SMEM_FULL_MIN = 152 * 1024, TS_SMEM_FULL_MAX = 226 * 1024;

struct TsArgs {
    const uint32_t* qt;
    const uint32_t* st;
    void* out;
    int m, n, k;
    int out_f16;
    int m_tiles, n_tiles;
    int tok;             // tokens per tile = MMA N (multiple of 16)
    int nrb_w;           // 16-row blocks of the resident matrix (tile pitch)
    int ksplit;
    int raw_stages, x_stages, a_stages;
    int teams;           // of expanding warps; raw_stages and a_stages are multiples of it
    int tmem_cols;
    int off_x, off_bars; // byte offsets in dynamic shared memory (1024-byte aligned base)
    int off_stage;       // grouped: results of a tile on their way out
    int off_push;        // where the other splits' sums come in (ts_pushes); 0: the splits read each other's rings
    int pdl;
    float out_mul;
    uint32_t fma_add, fma_mul;   // (20 - E) << 26 | (24 - E) << 10 and the pair (-8 * 2^-E, -8 * 2^-E) (Dec::fma_shift)
    int* status;
    // grouped (MoE) mode: token tiles come from a device table, one expert's weights (n rows) per tile; tok is then the most
    // rows that a tile holds
    const int* tile_expert;
    const int* tile_row0;
    const int* tile_rows;
    const int* num_tiles;
    int expert0;
    const float* row_w;  // optional factor per sorted row
    int glu;             // 1: interleaved gate / up row blocks; stores f16(silu(f16 gate) * f16 up), n / 2 values per row
    int tables_fresh;    // 1: a launch that may not be complete yet wrote the table: read it only after the dependency wait
};

__device__ __forceinline__ void umma_ts_f16(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accum)
        : "memory");
}
template <int GROUP, bool FMA, bool TEAMS>
__global__ void __launch_bounds__(ts_threads(TEAMS), 2)
gemm_ts_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_s, const TsArgs a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    constexpr int GPS = SK / GROUP;                                  // scale groups per stage: 1 or 4
    constexpr int EXP_WARPS = TEAMS ? TS_MAX_TEAMS * TS_TEAM : DQ_WARPS, ARRIVE = TEAMS ? TS_TEAM : DQ_WARPS;
    constexpr uint32_t RAW_STAGE = RAW_BYTES + ts_scale_bytes(GROUP);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // known to be warp-uniform
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
    const int NR = a.raw_stages, NX = a.x_stages, NA = a.a_stages;
    const int N = a.tok;
    const uint32_t x_half = (uint32_t)N * (BK * 2);                  // one k-block of the token tile
    auto raw_addr = [&](int s) { return base + (uint32_t)s * RAW_STAGE; };
    auto x_addr = [&](int s) { return base + (uint32_t)a.off_x + (uint32_t)s * (2 * x_half); };
    const uint32_t bars = base + (uint32_t)a.off_bars;
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_free = [&](int s) { return bars + 8u * (NR + s); };
    auto x_full = [&](int s) { return bars + 8u * (2 * NR + s); };
    auto x_free = [&](int s) { return bars + 8u * (2 * NR + NX + s); };
    auto a_ready = [&](int s) { return bars + 8u * (2 * NR + 2 * NX + s); };
    auto a_free = [&](int s) { return bars + 8u * (2 * NR + 2 * NX + NA + s); };
    const uint32_t accum_bar = bars + 8u * (2 * NR + 2 * NX + 2 * NA);

    // ---- this CTA's tile ----
    const int tile = (int)blockIdx.x, ks = a.ksplit, split = (int)blockIdx.y;
    const int ntile = a.m_tiles == 1 ? tile : tile / a.m_tiles, mtile = tile - ntile * a.m_tiles;    // neighbours share the weights
    const int n0 = ntile * TS_MROWS;
    const int m0 = mtile * N, rb0 = n0 / TILE_ROWS;
    const int rows_valid = min(N, a.m - m0);
    const int nrbv = min(TS_MROWS, a.n - n0) / TILE_ROWS;       // valid 16-row blocks
    const uint32_t kb_bytes = (uint32_t)nrbv * (TILE_WORDS * 4);
    // K range of this split in stages; the last stage of the matrix may hold one k-block (32-channel groups)
    const int nkb_all = a.k / BK, st_all = (nkb_all + 1) / 2;
    const int st0 = (int)((unsigned)(st_all * split) / (unsigned)ks);
    const int nst = (int)((unsigned)(st_all * (split + 1)) / (unsigned)ks) - st0;
    auto stage_kbs = [&](int it) { return min(2, nkb_all - 2 * (st0 + it)); };
    auto issue_raw = [&](int it, int s) {
        const int kbs = stage_kbs(it);
        mbar_expect_tx(raw_full(s), kbs * kb_bytes + ts_scale_bytes(GROUP));         // (scales past the end: zeros)
        tma_load_2d(raw_addr(s) + RAW_BYTES, &tmap_s, (st0 + it) * GPS * 8, rb0, raw_full(s));
        const uint32_t* src = a.qt + ((size_t)(2 * (st0 + it)) * a.nrb_w + rb0) * TILE_WORDS;
        bulk_load(raw_addr(s), src, kb_bytes, raw_full(s));
        if (kbs == 2) {
            bulk_load(raw_addr(s) + RAW_BYTES / 2, src + (size_t)a.nrb_w * TILE_WORDS, kb_bytes, raw_full(s));
        }
    };

    if (warp == 2 + EXP_WARPS) {
        // The warp that streams the weights makes the barriers, a lane each, and requests its first stages.  By one thread that also did the rest, one after the
        // other, the first weights were requested 2.3 us after the start (code that runs once is fetched as it runs); 7168 x 5120, 27 tokens, before and now:
        // 9.9 and 9.4 us, with the sums sent 9.1.
        if (lane == 0) {
            s_abort = 0;
        }
        for (int i = lane; i < 2 * (NR + NX + NA) + 1; i += 32) {
            const bool all = (i >= NR && i < 2 * NR) || (i >= 2 * (NR + NX) && i < 2 * (NR + NX) + NA);     // raw_free, a_ready
            mbar_init(bars + 8u * i, all ? ARRIVE : 1);
        }
        mbar_init_fence();
        __syncwarp();
        if (elect_one()) {
            // the weights do not depend on the previous kernel of the stream
            for (int it = 0; it < NR && it < nst; ++it) {
                issue_raw(it, it);
            }
        }
        __syncwarp();
    }
    if (ks > 1) {
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // waited for before the splits' sums: every CTA has started
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(a.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    const uint32_t tmem_a = tmem + (uint32_t)N;                      // A ring: [stage][64 columns]
    volatile int* abort_flag = &s_abort;

    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------------ tokens
        if (a.pdl) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            // Only now.  CTAs of the next kernel that came before this one holds its TMEM could take it and then wait for this kernel; and those that come
            // while the previous kernel still has its SMs pile up on the few that neither holds (68 row tiles in clusters of 2, 5120 channels, 48 tokens, in a
            // row: 11.5 to 13.2 us a launch, and 10.4).
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        }
        const bool leader = elect_one();
        int sx = 0, px = 1;
        for (int it = 0; it < nst; ++it) {
            if (it >= NX && !__all_sync(0xffffffffu, mbar_wait(x_free(sx), px, abort_flag, a.status, (31 << 16) | it))) {
                break;
            }
            if (leader) {
                // both k-blocks in one box (the second one of the last stage may lie outside: zeros)
                mbar_expect_tx(x_full(sx), 2 * x_half);
                tma_load_3d(x_addr(sx), &tmap_x, 0, m0, 2 * (st0 + it), x_full(sx));
            }
            __syncwarp();
            if (++sx == NX) {
                sx = 0;
                px ^= 1;
            }
        }
    } else if (warp == 2 + EXP_WARPS) {
        // ------------------------------------------------------------------ weights
        const bool leader = elect_one();
        int sr = 0, pr = 0;
        for (int it = NR; it < nst; ++it) {
            if (!__all_sync(0xffffffffu, mbar_wait(raw_free(sr), pr, abort_flag, a.status, (32 << 16) | it))) {
                break;
            }
            if (leader) {
                issue_raw(it, sr);
            }
            __syncwarp();
            if (++sr == NR) {
                sr = 0;
                pr ^= 1;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(TS_MROWS >> 4) << 24);
        const bool leader = elect_one();
        int sx = 0, px = 0, sa = 0, pa = 0;
        for (int it = 0; it < nst; ++it) {
            const bool in = mbar_wait(x_full(sx), px, abort_flag, a.status, (33 << 16) | it) &&
                            mbar_wait(a_ready(sa), pa, abort_flag, a.status, (34 << 16) | it);
            if (!__all_sync(0xffffffffu, in)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t db = umma_desc(x_addr(sx));
            const uint64_t db1 = db + (x_half >> 4);
            const uint32_t ta = tmem_a + (uint32_t)(sa * A_COLS);
            const bool two = stage_kbs(it) == 2;
            if (leader) {
#pragma unroll
                for (int j = 0; j < BK / 16; ++j) {
                    umma_ts_f16(tmem, ta + j * 8, db + 2 * j, idesc, (it > 0 || j > 0) ? 1u : 0u);
                }
                if (two) {
#pragma unroll
                    for (int j = 0; j < BK / 16; ++j) {
                        umma_ts_f16(tmem, ta + BK / 2 + j * 8, db1 + 2 * j, idesc, 1u);
                    }
                }
                umma_commit(a_free(sa));
                umma_commit(x_free(sx));
            }
            __syncwarp();
            if (++sx == NX) {
                sx = 0;
                px ^= 1;
            }
            if (++sa == NA) {
                sa = 0;
                pa ^= 1;
            }
        }
        if (ok && leader) {
            umma_commit(accum_bar);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ expand: raw int4 -> f16 in TMEM
        if (TEAMS) {
            // A team of four warps takes a stage, the teams take stages in turn (ts_expand_stage).
            const int quad = warp & 3, team = (warp - 2) >> 2, teams = a.teams;
            const uint32_t t_st = tmem_a + ((uint32_t)(quad * 32) << 16);
            int sr = team, sa = team;
            uint32_t pr = 0, pa = 1;
            for (int it = team; team < teams && it < nst; it += teams) {
                // (a warp leaves as a whole: an expired wait may be seen by some of its lanes first)
                const bool in = ts_expand_stage<GROUP, FMA>(
                    raw_addr(sr), quad, nrbv, lane, t_st + (uint32_t)(sa * A_COLS), a.fma_add, a.fma_mul,
                    [&]() { return __all_sync(0xffffffffu, mbar_wait(raw_full(sr), pr, abort_flag, a.status, (35 << 16) | it)) != 0; },
                    [&]() { return it < NA || __all_sync(0xffffffffu, mbar_wait(a_free(sa), pa, abort_flag, a.status, (36 << 16) | it)) != 0; },
                    [&]() { mbar_arrive(raw_free(sr)); }, [&]() { mbar_arrive(a_ready(sa)); });
                if (!in) {
                    ok = false;
                    break;
                }
                if ((sr += teams) >= NR) {
                    sr = team;
                    pr ^= 1;
                }
                if ((sa += teams) >= NA) {
                    sa = team;
                    pa ^= 1;
                }
            }
        } else {
            // One 16-row block per warp; a warp may touch the TMEM lanes 32 * (warp % 4) .. +31 = two row blocks.
            const int quad = warp & 3, half = (warp - 2) >> 2;
            const int rb = quad * 2 + half;
            const bool live = rb < nrbv;
            const int rbl = live ? rb : 0;
            const uint32_t t_st = tmem_a + ((uint32_t)(quad * 32 + half * 16) << 16);
            const uint32_t r_ld = base + (uint32_t)rbl * (TILE_WORDS * 4) + (uint32_t)lane * 16u;
            const uint32_t s_ld = base + (uint32_t)(RAW_BYTES + rbl * (GPS * 32)) + (uint32_t)(lane >> 2) * 4u;   // scale pairs of the lane's rows
            int sr = 0, pr = 0, sa = 0, pa = 1;
            for (int it = 0; it < nst; ++it) {
                // (a warp leaves as a whole: an expired wait may be seen by some of its lanes first)
                if (!__all_sync(0xffffffffu, mbar_wait(raw_full(sr), pr, abort_flag, a.status, (35 << 16) | it))) {
                    ok = false;
                    break;
                }
                const uint32_t ra = r_ld + (uint32_t)sr * RAW_STAGE;
                const uint4 raw0 = lds128(ra);
                const uint4 raw1 = lds128(ra + RAW_BYTES / 2);           // stale bytes when the stage holds one k-block
                uint32_t sc[GPS];
#pragma unroll
                for (int i = 0; i < GPS; ++i) {
                    sc[i] = lds32(s_ld + (uint32_t)sr * RAW_STAGE + (uint32_t)i * 32u);
                }
                uint32_t v[16];
                const TsScale<FMA> sc0(sc[0], a.fma_add, a.fma_mul), sc1(sc[GPS > 1 ? 1 : 0], a.fma_add, a.fma_mul);
                ts_expand<FMA>(raw0, sc0, sc1, v);
                if (it >= NA && !__all_sync(0xffffffffu, mbar_wait(a_free(sa), pa, abort_flag, a.status, (36 << 16) | it))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t td = t_st + (uint32_t)(sa * A_COLS);
                tmem_st_16x256b_x4(td, v);
                if (GPS > 1) {
                    ts_expand<FMA>(raw1, TsScale<FMA>(sc[GPS > 2 ? 2 : 0], a.fma_add, a.fma_mul), TsScale<FMA>(sc[GPS > 2 ? 3 : 0], a.fma_add, a.fma_mul), v);
                } else {
                    ts_expand<FMA>(raw1, sc0, sc1, v);
                }
                tmem_st_16x256b_x4(td + BK / 2, v);
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(raw_free(sr));                           // both k-blocks have been used (as in ts_expand_stage)
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(a_ready(sa));
                }
                if (++sr == NR) {
                    sr = 0;
                    pr ^= 1;
                }
                if (++sa == NA) {
                    sa = 0;
                    pa ^= 1;
                }
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        ok = ok && mbar_wait(accum_bar, 0, abort_flag, a.status, (37 << 16));
        ok = __all_sync(0xffffffffu, ok);
        if (a.pdl) {
            asm volatile("griddepcontrol.wait;" ::: "memory");       // outputs may be what the previous kernel still reads
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }

    // ---------------------------------------------------------------------- epilogue
    const bool dq_warp = warp >= 2 && warp < 2 + DQ_WARPS;           // (the third team has nothing to do with the results)
    const int quad = warp & 3, sub = (warp - 2) >> 2;
    constexpr int EW = DQ_WARPS / 4;                                 // warps that share a TMEM lane quadrant
    const int lrow = quad * 32 + lane;                               // weight row within the tile
    if (ks == 1 && a.out_f16) {
        // f16 results meet in shared memory ([token][row], the rings are idle) and leave as whole 16-byte pieces of a token's
        // row: a lane holds one weight row, so from registers it would store 2 bytes at a time (197 x 34816 x 5120: 62.9 -> 60.7
        // us; 64 tokens 32.2 -> 31.8)
        constexpr int PER_TOK = TS_MROWS * 2;
        if (dq_warp && ok) {
            for (int c0 = sub * 16; c0 < rows_valid; c0 += EW * 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    *reinterpret_cast<__half*>(base_ptr + (c0 + i) * PER_TOK + lrow * 2) = __float2half_rn(__uint_as_float(v[i]) * a.out_mul);
                }
            }
        }
        __syncthreads();
        if (!*abort_flag) {
            const int pieces = min(TS_MROWS, a.n - n0) / 8;
            __half* out = reinterpret_cast<__half*>(a.out) + (size_t)m0 * a.n + n0;
            for (int e = (int)threadIdx.x; e < rows_valid * pieces; e += ts_threads(TEAMS)) {
                const int tok = e / pieces, c = e - tok * pieces;
                *reinterpret_cast<uint4*>(out + (size_t)tok * a.n + c * 8) = *reinterpret_cast<const uint4*>(base_ptr + tok * PER_TOK + c * 16);
            }
        }
    } else if (ks == 1) {
        if (dq_warp && ok) {
            const bool row_ok = n0 + lrow < a.n;
            for (int c0 = sub * 16; c0 < rows_valid; c0 += EW * 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int tok = c0 + i;
                    if (tok < rows_valid && row_ok) {
                        reinterpret_cast<float*>(a.out)[(size_t)(m0 + tok) * a.n + n0 + lrow] = __uint_as_float(v[i]) * a.out_mul;
                    }
                }
            }
        }
    } else if (a.off_push > 0) {
        // Few tokens: a lane sends its row's sums to the CTA of the cluster that owns the row, into a place of their own beside the rings, and an
        // owner adds up what it has got, in split order: one barrier, no remote reads to wait for, and nobody to wait for before
        // leaving.
        const uint32_t rp = (uint32_t)(TS_MROWS + ks - 1) / (unsigned)ks, pitch = (uint32_t)ts_push_pitch(N);   // rows of an owner, at most; floats of a row
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (dq_warp && ok) {
            const uint32_t owner = (unsigned)(lrow * ks) / TS_MROWS, first = (owner * TS_MROWS + ks - 1) / (unsigned)ks;
            uint32_t there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(base + (uint32_t)a.off_push + ((uint32_t)split * rp + lrow - first) * pitch * 4u), "r"(owner));
            for (int c0 = sub * 16; c0 < rows_valid; c0 += EW * 16) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(there + (uint32_t)(c0 + i) * 4u), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]) : "memory");
                }
            }
        }
        cluster_sync_all();
        const int r0 = (split * TS_MROWS + ks - 1) / ks, rows = min(((split + 1) * TS_MROWS + ks - 1) / ks, a.n - n0) - r0;
        for (int tok = warp * 4; tok < rows_valid; tok += ts_threads(TEAMS) / 8) {       // a warp takes four tokens, a lane a row
            for (int r = lane; r < rows; r += 32) {
                const uint32_t q = base + (uint32_t)a.off_push + ((uint32_t)r * pitch + tok) * 4u;
                float4 sum = lds_f32x4(q);
                for (int i = 1; i < ks; ++i) {
                    const float4 v = lds_f32x4(q + (uint32_t)i * rp * pitch * 4u);
                    sum.x += v.x;
                    sum.y += v.y;
                    sum.z += v.z;
                    sum.w += v.w;
                }
                const float out[4] = {sum.x * a.out_mul, sum.y * a.out_mul, sum.z * a.out_mul, sum.w * a.out_mul};
                const size_t o = (size_t)(m0 + tok) * a.n + n0 + r0 + r;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (tok + i < rows_valid) {
                        if (a.out_f16) {
                            reinterpret_cast<__half*>(a.out)[o + (size_t)i * a.n] = __float2half_rn(out[i]);
                        } else {
                            reinterpret_cast<float*>(a.out)[o + (size_t)i * a.n] = out[i];
                        }
                    }
                }
            }
        }
    } else {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        // the splits' accumulators meet in distributed shared memory, RED_TOK tokens at a time: [token][row] f32 over the
        // (idle) rings; every CTA of the cluster adds an equal share of the elements over all splits, in split order
        constexpr int ROWS = TS_MROWS;
        for (int cb = 0; cb < rows_valid; cb += RED_TOK) {
            const int nt = min(RED_TOK, rows_valid - cb);
            if (dq_warp && ok) {
                for (int c0 = sub * 16; c0 < nt; c0 += EW * 16) {
                    uint32_t v[16];
                    tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cb + c0), v);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        *reinterpret_cast<float*>(base_ptr + ((c0 + i) * ROWS + lrow) * 4) = __uint_as_float(v[i]);
                    }
                }
            }
            cluster_sync_all();
            const int nr4 = min(ROWS, a.n - n0) / 4;
            const int total = nt * nr4;
            const int e0 = (int)((unsigned)(total * split) / (unsigned)ks), e1 = (int)((unsigned)(total * (split + 1)) / (unsigned)ks);
            for (int e = e0 + (int)threadIdx.x; e < e1; e += ts_threads(TEAMS)) {
                const int tok = e / nr4, r = (e - tok * nr4) * 4;
                float4 pv[8];
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    pv[s] = s < ks ? ld_dsmem_f32x4(base + (uint32_t)((tok * ROWS + r) * 4), (unsigned)s) : make_float4(0, 0, 0, 0);
                }
                float4 sum = pv[0];
#pragma unroll
                for (int s = 1; s < 8; ++s) {
                    if (s < ks) {
                        sum.x += pv[s].x;
                        sum.y += pv[s].y;
                        sum.z += pv[s].z;
                        sum.w += pv[s].w;
                    }
                }
                sum.x *= a.out_mul;
                sum.y *= a.out_mul;
                sum.z *= a.out_mul;
                sum.w *= a.out_mul;
                const size_t o = (size_t)(m0 + cb + tok) * a.n + n0 + r;
                if (a.out_f16) {
                    const __half2 h0 = __floats2half2_rn(sum.x, sum.y), h1 = __floats2half2_rn(sum.z, sum.w);
                    *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(a.out) + o) =
                        make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
                } else {
                    *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + o) = sum;
                }
            }
            cluster_sync_all();   // before the buffer is filled again, and before any CTA of the cluster leaves
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
    }
}


// Grouped (MoE) form: token tiles from a device table, one expert's weights per tile, persistent CTAs.  The roles are those of the dense
// kernel, but run on from tile to tile: with a CTA per tile, entry, table, TMEM, barriers and the first loads took about 4 us of the 14
// (K = 2048) or 8 (K = 768) that a tile of 128 experts x 2048 x 768 took.  Now the rings run ahead into the next tile while the last one is
// converted, and the two CTAs of an SM fill each other's epilogues.  (Layer of 128 experts, top-8: 256 tokens 165 ->
// 141 us, 1024 tokens 209 -> 186.)
template <int GROUP>
__global__ void __launch_bounds__(TSG_THREADS, 2)
gemm_ts_grouped_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_s, const TsArgs a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    constexpr int GPS = SK / GROUP;                                  // scale groups per stage: 1 or 4
    constexpr uint32_t RAW_STAGE = RAW_BYTES + ts_scale_bytes(GROUP);
    if (a.tables_fresh) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
    const int NR = a.raw_stages, NX = a.x_stages, NA = a.a_stages;
    const uint32_t x_half = (uint32_t)a.tok * (BK * 2);
    auto raw_addr = [&](int s) { return base + (uint32_t)s * RAW_STAGE; };
    auto x_addr = [&](int s) { return base + (uint32_t)a.off_x + (uint32_t)s * (2 * x_half); };
    const uint32_t bars = base + (uint32_t)a.off_bars;
    auto raw_full = [&](int s) { return bars + 8u * s; };
    auto raw_free = [&](int s) { return bars + 8u * (NR + s); };
    auto x_full = [&](int s) { return bars + 8u * (2 * NR + s); };
    auto x_free = [&](int s) { return bars + 8u * (2 * NR + NX + s); };
    auto a_ready = [&](int s) { return bars + 8u * (2 * NR + 2 * NX + s); };
    auto a_free = [&](int s) { return bars + 8u * (2 * NR + 2 * NX + NA + s); };
    const uint32_t accum_bar = bars + 8u * (2 * NR + 2 * NX + 2 * NA), acc_free = accum_bar + 8u;

    const int nkb = a.k / BK, nst = (nkb + 1) / 2;                   // the last stage may hold one k-block (32-channel groups)
    const int tiles = *a.num_tiles * a.n_tiles;
    // neighbours share the token rows, then the expert's weights
    struct Tile {
        int m0, rows, n0, rb0, nrbv;
    };
    auto tile_at = [&](int i) {
        const int mt = i / a.n_tiles;
        Tile r;
        r.n0 = (i - mt * a.n_tiles) * TS_MROWS;
        r.m0 = a.tile_row0[mt];
        r.rows = a.tile_rows[mt];
        r.rb0 = ((a.tile_expert[mt] - a.expert0) * a.n + r.n0) / TILE_ROWS;
        r.nrbv = min(TS_MROWS, a.n - r.n0) / TILE_ROWS;
        return r;
    };

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < NR; ++s) {
            mbar_init(raw_full(s), 1);
            mbar_init(raw_free(s), DQ_WARPS);
        }
        for (int s = 0; s < NX; ++s) {
            mbar_init(x_full(s), 1);
            mbar_init(x_free(s), 1);
        }
        for (int s = 0; s < NA; ++s) {
            mbar_init(a_ready(s), DQ_WARPS);
            mbar_init(a_free(s), 1);
        }
        mbar_init(accum_bar, 1);
        mbar_init(acc_free, DQ_WARPS);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(a.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // only now: a CTA of the next kernel that came earlier could take the TMEM this one still has to allocate
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    const uint32_t tmem_a = tmem + (uint32_t)a.tok;                  // A ring: [stage][64 columns]
    volatile int* abort_flag = &s_abort;

    // After a wait that ran out a role goes on through its loops without waiting, loading or multiplying, so that the barrier of the
    // converting warps stays matched.
    bool ok = true;
    if (warp == 0) {
        // ------------------------------------------------------------------ tokens
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const bool leader = elect_one();
        int sx = 0;
        uint32_t px = 1, cnt = 0;
        for (int i = blockIdx.x; i < tiles && ok; i += gridDim.x) {
            const Tile tl = tile_at(i);
            const int boxes = (tl.rows + TS_XBOX - 1) / TS_XBOX;     // rows of the next expert, or zeros, fill the last box up
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)NX && !__all_sync(0xffffffffu, mbar_wait(x_free(sx), px, abort_flag, a.status, (51 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    const int kbs = min(2, nkb - 2 * it);
                    mbar_expect_tx(x_full(sx), (uint32_t)(kbs * boxes) * (TS_XBOX * BK * 2));
                    for (int h = 0; h < kbs; ++h) {
                        for (int c = 0; c < boxes; ++c) {
                            tma_load_2d(x_addr(sx) + h * x_half + (uint32_t)c * (TS_XBOX * BK * 2), &tmap_x, (2 * it + h) * BK,
                                        tl.m0 + c * TS_XBOX, x_full(sx));
                        }
                    }
                }
                __syncwarp();
                if (++sx == NX) {
                    sx = 0;
                    px ^= 1;
                }
            }
        }
    } else if (warp == 2 + DQ_WARPS) {
        // ------------------------------------------------------------------ weights (they do not depend on the previous kernel)
        const bool leader = elect_one();
        int sr = 0;
        uint32_t pr = 1, cnt = 0;
        for (int i = blockIdx.x; i < tiles && ok; i += gridDim.x) {
            const Tile tl = tile_at(i);
            const uint32_t kb_bytes = (uint32_t)tl.nrbv * (TILE_WORDS * 4);
            for (int it = 0; it < nst; ++it, ++cnt) {
                if (cnt >= (uint32_t)NR && !__all_sync(0xffffffffu, mbar_wait(raw_free(sr), pr, abort_flag, a.status, (52 << 16) | it))) {
                    ok = false;
                    break;
                }
                if (leader) {
                    const int kbs = min(2, nkb - 2 * it);
                    mbar_expect_tx(raw_full(sr), kbs * kb_bytes + ts_scale_bytes(GROUP));
                    tma_load_2d(raw_addr(sr) + RAW_BYTES, &tmap_s, it * GPS * 8, tl.rb0, raw_full(sr));
                    const uint32_t* src = a.qt + ((size_t)(2 * it) * a.nrb_w + tl.rb0) * TILE_WORDS;
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
        int sx = 0, sa = 0;
        uint32_t px = 0, pa = 0, done = 0;
        for (int i = blockIdx.x; i < tiles && ok; i += gridDim.x, ++done) {
            const int rows = a.tile_rows[i / a.n_tiles];
            const uint32_t idesc = (1u << 4) | ((uint32_t)((rows + 15) / 16 * 2) << 17) | ((uint32_t)(TS_MROWS >> 4) << 24);
            // the accumulator is read before it is written again
            if (done > 0 && !__all_sync(0xffffffffu, mbar_wait(acc_free, (done - 1) & 1, abort_flag, a.status, (53 << 16)))) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int it = 0; it < nst; ++it) {
                const bool in = mbar_wait(x_full(sx), px, abort_flag, a.status, (54 << 16) | it) &&
                                mbar_wait(a_ready(sa), pa, abort_flag, a.status, (55 << 16) | it);
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
                        umma_ts_f16(tmem, ta + j * 8, db + 2 * j, idesc, (it > 0 || j > 0) ? 1u : 0u);
                    }
                    if (two) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) {
                            umma_ts_f16(tmem, ta + BK / 2 + j * 8, db1 + 2 * j, idesc, 1u);
                        }
                    }
                    umma_commit(a_free(sa));
                    umma_commit(x_free(sx));
                    if (it + 1 == nst) {
                        umma_commit(accum_bar);
                    }
                }
                __syncwarp();
                if (++sx == NX) {
                    sx = 0;
                    px ^= 1;
                }
                if (++sa == NA) {
                    sa = 0;
                    pa ^= 1;
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ expand: raw int4 -> f16 in TMEM; then convert and store
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const int rb = quad * 2 + half;                              // a warp may touch the TMEM lanes 32 * (warp % 4) .. +31
        const int lrow = quad * 32 + lane;
        const int et = (int)threadIdx.x - 64;                        // thread among the converting warps
        const bool glu = a.glu != 0;
        const int per_tok = glu ? TS_MROWS : TS_MROWS * 2, n_out = glu ? a.n / 2 : a.n;      // bytes; values per row of the result
        unsigned char* stage_ptr = base_ptr + a.off_stage;
        const uint32_t t_st = tmem_a + ((uint32_t)(quad * 32 + half * 16) << 16);
        int sr = 0, sa = 0;
        uint32_t pr = 0, pa = 1, cnt = 0, done = 0;
        Tile tl{}, next{};
        if ((int)blockIdx.x < tiles) {
            next = tile_at(blockIdx.x);
        }
        for (int i = blockIdx.x; i < tiles; i += gridDim.x, ++done) {
            tl = next;
            const bool more = i + (int)gridDim.x < tiles;
            if (more) {
                next = tile_at(i + (int)gridDim.x);
            }
            const int rbl = rb < tl.nrbv ? rb : 0;
            const uint32_t r_ld = base + (uint32_t)rbl * (TILE_WORDS * 4) + (uint32_t)lane * 16u;
            const uint32_t s_ld = base + (uint32_t)(RAW_BYTES + rbl * (GPS * 32)) + (uint32_t)(lane >> 2) * 4u;
            for (int it = 0; it < nst && ok; ++it, ++cnt) {
                if (!__all_sync(0xffffffffu, mbar_wait(raw_full(sr), pr, abort_flag, a.status, (56 << 16) | it))) {
                    ok = false;
                    break;
                }
                const uint32_t ra = r_ld + (uint32_t)sr * RAW_STAGE;
                const uint4 raw0 = lds128(ra);
                const uint4 raw1 = lds128(ra + RAW_BYTES / 2);       // stale bytes when the stage holds one k-block
                uint32_t sc[GPS];
#pragma unroll
                for (int q = 0; q < GPS; ++q) {
                    sc[q] = lds32(s_ld + (uint32_t)sr * RAW_STAGE + (uint32_t)q * 32u);
                }
                uint32_t v[16];
                ts_expand<false>(raw0, TsScale<false>(sc[0], 0, 0), TsScale<false>(sc[GPS > 1 ? 1 : 0], 0, 0), v);
                if (cnt >= (uint32_t)NA && !__all_sync(0xffffffffu, mbar_wait(a_free(sa), pa, abort_flag, a.status, (57 << 16) | it))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t td = t_st + (uint32_t)(sa * A_COLS);
                tmem_st_16x256b_x4(td, v);
                ts_expand<false>(raw1, TsScale<false>(sc[GPS > 2 ? 2 : 0], 0, 0), TsScale<false>(sc[GPS > 2 ? 3 : 0], 0, 0), v);
                tmem_st_16x256b_x4(td + BK / 2, v);
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(raw_free(sr));                       // both k-blocks have been used (as in ts_expand_stage)
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(a_ready(sa));
                }
                if (++sr == NR) {
                    sr = 0;
                    pr ^= 1;
                }
                if (++sa == NA) {
                    sa = 0;
                    pa ^= 1;
                }
            }
            ok = ok && mbar_wait(accum_bar, done & 1, abort_flag, a.status, (58 << 16));
            ok = __all_sync(0xffffffffu, ok);
            if (done == 0) {
                asm volatile("griddepcontrol.wait;" ::: "memory");   // outputs may be what the previous kernel still reads
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // f16 results through shared memory, [token][row], a stage of 16 KB at a time
            const int stage_tok = TS_STAGE_BYTES / per_tok;
            for (int t0 = 0; t0 < tl.rows; t0 += stage_tok) {
                const int nt = min(stage_tok, tl.rows - t0);
                if (ok) {
                    for (int c0 = half * 16; c0 < nt; c0 += 32) {
                        uint32_t v[16];
                        tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(t0 + c0), v);
                        if (glu) {
                            // lanes 0-15 hold gate sums, lanes 16-31 the up sums of the same outputs: the former take tokens 0-7 of
                            // the chunk, the latter 8-15
                            const bool hi = lane >= 16;
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                const float mine = __uint_as_float(hi ? v[q + 8] : v[q]) * a.out_mul;
                                const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(hi ? v[q] : v[q + 8]), 16) * a.out_mul;
                                *reinterpret_cast<__half*>(stage_ptr + (c0 + q + (hi ? 8 : 0)) * per_tok + (quad * 16 + (lane & 15)) * 2) =
                                    silu_mul_f16(hi ? other : mine, hi ? mine : other);
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < 16; ++q) {
                                float f = __uint_as_float(v[q]) * a.out_mul;
                                if (a.row_w != nullptr) {
                                    f = mul_row_w(f, c0 + q < nt ? a.row_w[tl.m0 + t0 + c0 + q] : 0.f);
                                }
                                *reinterpret_cast<__half*>(stage_ptr + (c0 + q) * per_tok + lrow * 2) = __float2half_rn(f);
                            }
                        }
                    }
                }
                if (t0 + stage_tok >= tl.rows) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(acc_free);
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"n"(DQ_WARPS * 32) : "memory");
                if (ok) {
                    const int pieces = min(TS_MROWS, a.n - tl.n0) / (glu ? 16 : 8);
                    __half* out = reinterpret_cast<__half*>(a.out) + (size_t)(tl.m0 + t0) * n_out + (glu ? tl.n0 / 2 : tl.n0);
                    for (int e = et; e < nt * pieces; e += DQ_WARPS * 32) {
                        const int tok = e / pieces, c = e - tok * pieces;
                        *reinterpret_cast<uint4*>(out + (size_t)tok * n_out + c * 8) =
                            *reinterpret_cast<const uint4*>(stage_ptr + tok * per_tok + c * 16);
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"n"(DQ_WARPS * 32) : "memory");     // the stage is free again
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
    }
}

}  // namespace


// bytes of `nr` raw stages; what follows is 1024-byte aligned
static size_t ts_raw_bytes(int group, int nr) { return ((size_t)nr * (RAW_BYTES + ts_scale_bytes(group)) + 1023) & ~(size_t)1023; }

static size_t ts_smem(int group, int tok, int nr, int nx, int na, int* off_x, int* off_bars) {
    size_t off = ts_raw_bytes(group, nr);
    *off_x = (int)off;
    off += (size_t)nx * tok * SK * 2;
    const size_t red = (size_t)std::min(RED_TOK, tok) * TS_MROWS * 4;   // the cluster's sum reuses the rings
    off = std::max(off, red);
    *off_bars = (int)off;
    return off + (size_t)(2 * nr + 2 * nx + 2 * na + 1) * 8 + 1024;
}

cudaError_t gemm_ts_init_device() {
    cudaError_t e = cudaSuccess;
    for (const void* f : {(const void*)gemm_ts_kernel<128, false, false>, (const void*)gemm_ts_kernel<128, true, false>, (const void*)gemm_ts_kernel<32, false, false>,
                          (const void*)gemm_ts_kernel<128, false, true>, (const void*)gemm_ts_kernel<128, true, true>, (const void*)gemm_ts_kernel<32, false, true>,
                          (const void*)gemm_ts_grouped_kernel<128>, (const void*)gemm_ts_grouped_kernel<32>}) {
        if (e == cudaSuccess) {
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TS_SMEM_FULL_MAX);
        }
    }
    return e;
}

// Shared memory and ring depths of a launch with tiles of `tok` tokens.
namespace {
struct TsPlan {
    int tmem_cols, na, nr, nx, off_x, off_bars, off_push;
    int teams;           // 0: a warp per row block
    size_t smem;
};
TsPlan ts_plan(int group, int tok, bool teams, int ks) {
    TsPlan p{};
    // TMEM: the accumulator and as many expanded stages as fit in half of it (two CTAs per SM), else in all of it
    p.tmem_cols = tok <= 128 ? 256 : 512;
    p.na = std::min((p.tmem_cols - tok) / A_COLS, 4);
    const size_t push = ts_pushes(tok, ks) ? (size_t)ks * ((TS_MROWS + ks - 1) / ks) * ts_push_pitch(tok) * 4 + 16 : 0;
    const size_t limit = (p.tmem_cols == 256 ? TS_SMEM_HALF_MAX : TS_SMEM_FULL_MAX) - push;
    p.teams = !teams ? 0 : p.na % 3 == 0 ? 3 : 2;
    const int step = std::max(1, p.teams);                       // the rings divide by the teams
    p.nx = p.nr = ts_smem(group, tok, 3, 3, p.na, &p.off_x, &p.off_bars) <= limit ? 3 : 2;
    p.nr = (p.nr + step - 1) / step * step;
    while (p.nr + step <= 12 && ts_smem(group, tok, p.nr + step, p.nx, p.na, &p.off_x, &p.off_bars) <= limit) {
        p.nr += step;
        if ((teams || p.nr % 2 == 0) && p.nx < 4 && ts_smem(group, tok, p.nr, p.nx + 1, p.na, &p.off_x, &p.off_bars) <= limit) {
            ++p.nx;
        }
    }
    const size_t used = ts_smem(group, tok, p.nr, p.nx, p.na, &p.off_x, &p.off_bars);
    p.off_push = push > 0 ? (p.off_bars + (2 * (p.nr + p.nx + p.na) + 1) * 8 + 15) & ~15 : 0;
    p.smem = std::max(used + push, p.tmem_cols == 256 ? TS_SMEM_HALF_MIN : TS_SMEM_FULL_MIN);
    return p;
}
}  // namespace

// Clusters of `ks` CTAs that can be resident at once, for half- and full-TMEM CTAs.  A cluster lies within a GPC, so large
// clusters leave room unused.  Two half-TMEM CTAs fit on an SM, and at least twice the clusters of whole-SM CTAs with them:
// the occupancy query counts one per SM, but 56 clusters of 4 run as one wave (27 x 7168 x 5120: 11.2 us against 13.3 with
// 2) and 40 of 6 too (27 x 5120 x 17408: 20.3 against 30.3 us with 3).
void Dec::ts_query_clusters() {
    for (int ks = 1; ks <= TS_MAX_SPLIT; ++ks) {
        int n = sm_count;
        if (ks > 1) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(1, ks);
            cfg.blockDim = dim3(ts_threads(false));
            cfg.dynamicSmemBytes = TS_SMEM_FULL_MAX;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1;
            attr[0].val.clusterDim.y = ks;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_ts_kernel<128, false, false>, &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;       // then this split is not considered
            }
        }
        ts_clusters[1][ks] = n;
        ts_clusters[0][ks] = 2 * n;
    }
}

// Tokens per tile and K split with the least estimated time (microseconds, fitted to measurements on B200): 3 us per launch;
// a stage of 128 channels takes 0.48 us and 0.0006 per token when the CTA has its SM alone (wide tiles more when all SMs run:
// 0.82 at 256 tokens) and 0.65 us and 0.0018 per token with a second one beside it; a split CTA another 1.2 us and 0.04 us per
// token for the sum over the cluster.  Without a candidate (a cluster size that is asked for and cannot be resident) the result
// has tok = 0 and a cost above every other form's.
TsChoice Dec::gemm_ts_choose(int n, int k, int t) const {
    TsChoice best{0, 0, 1e30};
    const int n_tiles = (n + TS_MROWS - 1) / TS_MROWS, stages = (k + SK - 1) / SK;
    int last_tok = 0;
    for (int cap : {256, 192, 128, 96, 64}) {
        const int m_tiles = (t + cap - 1) / cap;
        const int tok = ((t + m_tiles - 1) / m_tiles + 15) / 16 * 16;
        if (tok == last_tok || (tune_ts_tok > 0 && cap != tune_ts_tok)) {
            continue;
        }
        last_tok = tok;
        const long long tiles = (long long)m_tiles * n_tiles;
        const int full = tok > 128;
        for (int ks = 1; ks <= TS_MAX_SPLIT && ks <= stages; ++ks) {
            const int room = ts_clusters[full][ks];
            if (room <= 0 || (tune_ts_ks > 0 && ks != std::min(tune_ts_ks, stages))) {
                continue;
            }
            const double around = ks > 1 ? 1.2 + 0.04 * tok : 0.01 * tok;
            const int nst = (stages + ks - 1) / ks;
            auto stage = [&](long long ctas) {
                if (!full && ctas > sm_count) {
                    return 0.65 + 0.0018 * tok;
                }
                return 0.48 + 0.0006 * tok + (full && ctas > 128 ? 0.06 + 0.0020 * std::max(0, tok - 192) : 0.0);
            };
            const long long waves = tiles / room, rest = tiles - waves * room;
            double c = 3.0 + waves * (nst * stage((long long)room * ks) + around);
            if (rest > 0) {
                c += nst * stage(rest * ks) + around;
            }
            if (c < best.cost) {
                best = TsChoice{tok, ks, c};
            }
        }
    }
    return best;
}

int Dec::gemm_ts(const Lin* l, const void* x, void* dst, int t, int out_kind, const TsChoice& c, cudaStream_t st) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    // Teams where stages follow one another quickly: up to 64 tokens, to 96 with two CTAs on an SM.  A CTA of few stages has its first one sooner
    // with all warps on it (us, a warp per row block / teams: 27 x 34816 x 5120 27.2 / 25.6, groups of 32 31.0 / 28.9; 96 x 34816 x 5120 33.3 /
    // 29.2; 72 x 4096 x 4096 10.4 / 10.7, 197 x 5120 x 6144 21.2 / 22.0, 9 x 1024 x 1024 in clusters of 8 3.4 / 3.6).
    const long long ctas = (long long)((t + c.tok - 1) / c.tok) * ((l->n + TS_MROWS - 1) / TS_MROWS) * c.ks;
    const int nst = ((l->k + SK - 1) / SK + c.ks - 1) / c.ks;
    const bool teams = nst >= 4 && (c.tok <= 64 || (c.tok <= 96 && ctas > sm_count && nst >= 16));
    const TsPlan p = ts_plan(l->group, c.tok, teams, c.ks);
    TsArgs a{};
    a.tok = c.tok;
    a.ksplit = c.ks;
    a.m_tiles = (t + c.tok - 1) / c.tok;
    a.n_tiles = (l->n + TS_MROWS - 1) / TS_MROWS;
    a.tmem_cols = p.tmem_cols;
    a.a_stages = p.na;
    a.raw_stages = p.nr;
    a.teams = p.teams;
    a.x_stages = p.nx;
    a.off_x = p.off_x;
    a.off_bars = p.off_bars;
    a.off_push = p.off_push;
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)BK, (cuuint64_t)t, (cuuint64_t)(l->k / BK)};
    const cuuint64_t strides[2] = {(cuuint64_t)l->k * 2, (cuuint64_t)BK * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)a.tok, 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CUtensorMap smap;
    if (cr == CUDA_SUCCESS) {
        cr = ts_scale_map(enc, &smap, l->st, l->n, l->k, l->group);
    }
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
    cfg.gridDim = dim3(a.m_tiles * a.n_tiles, a.ksplit);
    cfg.blockDim = dim3(ts_threads(teams));
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (a.pdl) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    if (a.ksplit > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = 1;
        attr[n_attr].val.clusterDim.y = a.ksplit;
        attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    cudaError_t e;
    if (l->group != 128) {
        e = cudaLaunchKernelEx(&cfg, teams ? gemm_ts_kernel<32, false, true> : gemm_ts_kernel<32, false, false>, map, smap, a);
    } else if (l->fma_e < 0) {
        e = cudaLaunchKernelEx(&cfg, teams ? gemm_ts_kernel<128, false, true> : gemm_ts_kernel<128, false, false>, map, smap, a);
    } else {
        // one f16 operation per pair of weights where two do it otherwise, in the expansion that a small batch waits for (27 x 34816 x
        // 5120: 29.8 -> 26.5 us, 27 x 5120 x 17408: 21.3 -> 19.3); the weights come out 2^-E smaller
        const __half2 mul = __float2half2_rn(ldexpf(-8.0f, -l->fma_e));
        memcpy(&a.fma_mul, &mul, sizeof(mul));
        a.fma_add = ((uint32_t)(20 - l->fma_e) << 26) + ((uint32_t)(24 - l->fma_e) << 10);
        a.out_mul = ldexpf(l->out_mul, l->fma_e);
        e = cudaLaunchKernelEx(&cfg, teams ? gemm_ts_kernel<128, true, true> : gemm_ts_kernel<128, true, false>, map, smap, a);
    }
    if (e != cudaSuccess) {
        return cuda_fail("launch gemm", e);
    }
    last_kernel = "gemm_ts_kernel<" + std::to_string(l->group) + (l->fma_e >= 0 ? ",fma> " : "> ") + std::to_string(c.tok) + "-token tiles" +
                  (c.ks > 1 ? ", clusters of " + std::to_string(c.ks) : std::string());
    launches++;
    return 0;
}

// Grouped form over expert segments: `l` stacks the local experts along n (n_per_expert rows each); xs holds the gathered rows
// (sorted by expert), the token-tile table (at most `tok` rows each) lives on the device (moe.cu).
int Dec::gemm_ts_grouped(const Lin* l, const void* xs, int xs_rows, void* out, int n_per_expert, const MoeBufs& b, int max_tiles,
                         int tok, const float* row_w, cudaStream_t st, bool tables_fresh) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled is not available from the driver");
    }
    // half of the TMEM: the accumulator and as many expanded stages as fit; two CTAs per SM
    const int tmem_cols = 256, na = std::min((tmem_cols - tok) / A_COLS, 4), nx = tok <= 64 ? 3 : 2;
    TsArgs a{};
    int nr = 2;
    auto bars_at = [&](int raw) { return (int)ts_raw_bytes(l->group, raw) + nx * tok * SK * 2 + TS_STAGE_BYTES; };
    auto smem_of = [&](int raw) { return (size_t)bars_at(raw) + (size_t)(2 * raw + 2 * nx + 2 * na + 2) * 8 + 1024; };
    while (nr < 8 && smem_of(nr + 1) <= TS_SMEM_HALF_MAX) {
        ++nr;
    }
    a.tok = tok;
    a.ksplit = 1;
    a.m_tiles = max_tiles;
    a.n_tiles = (n_per_expert + TS_MROWS - 1) / TS_MROWS;
    a.tmem_cols = tmem_cols;
    a.a_stages = na;
    a.raw_stages = nr;
    a.x_stages = nx;
    a.off_x = (int)ts_raw_bytes(l->group, nr);
    a.off_stage = a.off_x + nx * tok * SK * 2;
    a.off_bars = bars_at(nr);
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)l->k, (cuuint64_t)xs_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)l->k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)TS_XBOX};
    const cuuint32_t estr[2] = {1, 1};
    CUresult cr = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(xs), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    CUtensorMap smap;
    if (cr == CUDA_SUCCESS) {
        cr = ts_scale_map(enc, &smap, l->st, l->n, l->k, l->group);
    }
    if (cr != CUDA_SUCCESS) {
        return fail("w4a16 gemm: cuTensorMapEncodeTiled failed (%d)", (int)cr);
    }
    a.qt = l->qt;
    a.st = (const uint32_t*)l->st;
    a.out = out;
    a.m = xs_rows;
    a.n = n_per_expert;
    a.k = l->k;
    a.out_f16 = 1;
    a.nrb_w = l->n / TILE_ROWS;
    a.pdl = tune_pdl ? 1 : 0;
    a.out_mul = l->out_mul;
    a.status = gemm_status;
    a.tile_expert = b.tile_expert;
    a.tile_row0 = b.tile_row0;
    a.tile_rows = b.tile_rows;
    a.num_tiles = b.n_tiles;
    a.expert0 = moe.e0;
    a.row_w = row_w;
    a.glu = l->glu_f > 0 ? 1 : 0;
    a.tables_fresh = tables_fresh ? 1 : 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min(a.m_tiles * a.n_tiles, 2 * sm_count));
    cfg.blockDim = dim3(TSG_THREADS);
    cfg.dynamicSmemBytes = std::max(smem_of(nr), TS_SMEM_HALF_MIN);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (a.pdl) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    const cudaError_t e = l->group == 128 ? cudaLaunchKernelEx(&cfg, gemm_ts_grouped_kernel<128>, map, smap, a)
                                          : cudaLaunchKernelEx(&cfg, gemm_ts_grouped_kernel<32>, map, smap, a);
    if (e != cudaSuccess) {
        return cuda_fail("launch grouped gemm", e);
    }
    last_kernel = "gemm_ts_grouped_kernel<" + std::to_string(l->group) + "> " + std::to_string(tok) + "-row tiles";
    launches++;
    return 0;
}

}  // namespace w4
