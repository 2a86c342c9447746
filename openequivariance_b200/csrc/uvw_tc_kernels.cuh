// "uvw" forward pass on the 5th-generation tensor cores (tcgen05, TMEM accumulators), FP32 in / FP32
// out with 3xTF32 error compensation, for shared weights and second-input multiplicity 1.
//
//   Z[b,o,w,k] = sum_{paths p -> o} sum_u W_p[u,w] * T_p[b,u,k],   T_p[b,u,k] = sum_{ij} C_p[i,j,k] x[b,u,i] y[b,j]
//
// is a GEMM whose A operand does not exist in memory: rows are (batch row, k), the K axis is (path, u),
// N is the output multiplicity.  Per output irrep o the CTA keeps W (split into TF32 "hi" and "lo"
// parts, pre-swizzled by oeq_uvw_pack_weights) resident in shared memory and walks its share of the
// batch in chunks of floor(128 / (2l+1)) rows:
//
//   * 16 producer warps form T with the Clebsch-Gordan constants unrolled, split every value into
//     hi = tf32(t), lo = tf32(t - hi), and store both as K-major 128-byte-swizzled [128 x 32] tiles;
//   * one warp issues tcgen05.mma (M = 128, N = mul_out, K = 8 per instruction) three times per K step
//     (hi.hi + hi.lo + lo.hi) into a ring of TMEM accumulator tiles, and hands shared-memory stages
//     and accumulators on with tcgen05.commit -> mbarrier;
//   * 4 epilogue warps read accumulators with tcgen05.ld, transpose (row,k)-major tiles through a
//     padded shared-memory buffer and write Z rows coalesced.
//
// Replaces the reference's per-row warp matmul (openequivariance/templates/wmm.cuh:1-88,
// openequivariance/templates/loop_unroll_tp.cuh:54-83).  Every wait is bounded; on expiry the role
// records a code in *status and stops, and the CTA still frees its tensor memory.
#pragma once
#include "oeq_common.cuh"
#include "tc_common.cuh"

namespace oeq {
using namespace oeqd;

struct UvwTcParams {
    const float* X;
    const float* Y;
    const float* Wpacked;   // output of oeq_uvw_pack_weights
    float* Z;
    long long batch;
    int* status;
    int dealt;                  // chunks of all output irreps dealt to the CTAs, instead of a share of the rows each
    unsigned long long* prof;   // optional cycle accounting of CTA 0 (development aid), else null
};

// Roles (macros from the host): TC_PW producer warps (8 or 16) and TC_EPI groups of four epilogue warps.  Forward pass:
// 16 and 1, since forming T bounds it.  The product W dZ of the backward pass (UNIT_Y): 8 and 2; its operand tiles are
// dZ itself and serve up to 256 columns, and writing dT bounds it.
constexpr int TC_PRODUCER_WARPS = TC_PW;
constexpr int TC_EPI_GROUPS = TC_EPI;
constexpr int TC_EPILOGUE_WARPS = 4;            // of one group
constexpr int TC_THREADS = (TC_PRODUCER_WARPS + 1 + TC_EPI_GROUPS * TC_EPILOGUE_WARPS) * 32;
constexpr int TC_NA = 2;                       // A-operand stages
constexpr int TC_STAGE_HALF = 128 * 128;       // one [128 rows x 32 tf32] swizzled tile
constexpr int TC_STAGE_BYTES = 2 * TC_STAGE_HALF;   // hi + lo
constexpr int ERR_TC_A_EMPTY = 11, ERR_TC_A_FULL = 12, ERR_TC_ACC_EMPTY = 13, ERR_TC_ACC_FULL = 14, ERR_TC_W = 15;

// ---- compile-time geometry ------------------------------------------------------------------
constexpr int tc_khalves(int p) { return (IN1_MUL[I_IN1[p]] + 31) / 32; }
constexpr int tc_blocks_before(int o, int p_end) {   // [MW x 32] weight blocks of output o before path p_end
    int n = 0;
    for (int p = 0; p < p_end; ++p)
        if (I_OUT[p] == o) n += tc_khalves(p);
    return n;
}
constexpr int tc_mwp(int o) { return (OUT_MUL[o] + 15) / 16 * 16; }              // N of the MMA: a multiple of 16
constexpr int tc_block_bytes(int o) { return tc_mwp(o) * 128; }                  // one hi (or lo) block
constexpr int tc_w_bytes(int o) { return tc_blocks_before(o, N_INSTR) * 2 * tc_block_bytes(o); }
constexpr int tc_w_offset(int o) {   // byte offset of output o inside the packed weight buffer
    int b = 0;
    for (int q = 0; q < o; ++q) b += tc_w_bytes(q);
    return b;
}
constexpr int tc_w_max() {
    int m = 0;
    for (int o = 0; o < N_OUT; ++o) m = tc_w_bytes(o) > m ? tc_w_bytes(o) : m;
    return m;
}
constexpr int tc_mw_max() {
    int m = 16;
    for (int o = 0; o < N_OUT; ++o) m = tc_mwp(o) > m ? tc_mwp(o) : m;
    return m;
}
constexpr bool tc_wide(int o) { return 2 * tc_mwp(o) <= 256; }
constexpr int tc_acc_cols(int o) { return tc_wide(o) ? 2 * tc_mwp(o) : tc_mwp(o); }
// One ring of accumulator tiles serves all output irreps: equal tile width and count for all of them, so that
// tile index and barrier phase follow from one running counter.
constexpr int tc_acc_cols_max() {
    int m = 16;
    for (int o = 0; o < N_OUT; ++o) m = tc_acc_cols(o) > m ? tc_acc_cols(o) : m;
    return m;
}
constexpr int TC_ACC_COLS = tc_acc_cols_max();
constexpr int TC_W_MAX = tc_w_max();
constexpr int TC_MW_MAX = tc_mw_max();
// An accumulator tile is drained in blocks of columns, dealt to the epilogue groups.
constexpr int TC_BLOCK_COLS = TC_EPI_GROUPS > 1 ? 32 : (TC_MW_MAX < 64 ? TC_MW_MAX : 64);
constexpr int TC_STG_PITCH = TC_BLOCK_COLS + 1;     // floats per staged accumulator row (odd: conflict free)
constexpr int TC_STG_BYTES = (128 * TC_STG_PITCH * 4 + 15) / 16 * 16;
constexpr int TC_TMEM_COLS = 512;

// shared memory map (1024-byte aligned base): [A stages][W of one output][epilogue staging][barriers]
constexpr int TC_OFF_A = 0;
constexpr int TC_OFF_W = TC_OFF_A + TC_NA * TC_STAGE_BYTES;
constexpr int TC_OFF_STG = TC_OFF_W + (TC_W_MAX + 1023) / 1024 * 1024;
constexpr int TC_OFF_BAR = TC_OFF_STG + TC_EPI_GROUPS * TC_STG_BYTES;
constexpr int TC_MAX_ACC = 32;
constexpr int TC_NACC = TC_TMEM_COLS / TC_ACC_COLS < TC_MAX_ACC ? TC_TMEM_COLS / TC_ACC_COLS : TC_MAX_ACC;
constexpr int TC_SMEM_BYTES = TC_OFF_BAR + (2 * TC_NA + 2 * TC_MAX_ACC + 2) * 8 + 16 + 1024;   // + alignment slack

struct TcBars {
    unsigned long long* a_full;     // [TC_NA]
    unsigned long long* a_empty;    // [TC_NA]
    unsigned long long* acc_full;   // [TC_MAX_ACC]
    unsigned long long* acc_empty;  // [TC_MAX_ACC]
    unsigned long long* w_full;
    unsigned long long* w_free;
    unsigned* tmem_slot;
    __device__ explicit TcBars(unsigned char* base) {
        unsigned long long* b = reinterpret_cast<unsigned long long*>(base + TC_OFF_BAR);
        a_full = b; a_empty = b + TC_NA; acc_full = b + 2 * TC_NA; acc_empty = acc_full + TC_MAX_ACC;
        w_full = acc_empty + TC_MAX_ACC; w_free = w_full + 1;
        tmem_slot = reinterpret_cast<unsigned*>(w_free + 1);
    }
};


// Batch rows of a chunk and the accumulator row of (batch row r, component k): k-major, with the rows rounded down to
// a multiple of eight where that costs at most an eighth of the tile.  A producer warp then keeps its row of the
// swizzle pattern (r mod 8) and every store of a stage has a compile-time offset.
constexpr int tc_rpc(int o) {
    const int full = 128 / OUT_D[o], r8 = full / 8 * 8;
    return r8 * OUT_D[o] >= 112 ? r8 : full;
}

constexpr int tc_first_path(int o) {
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o) return p;
    return 0;
}
// Relative time of a chunk of output o.  Forward: the producers, about one instruction per input and output component and
// coefficient and row, but no stage is shorter than its MMAs.  The product W dZ: draining its columns.
constexpr int tc_chunk_cost(int o) {
    int n = 16;
    for (int p = 0; p < N_INSTR; ++p) {
        if (I_OUT[p] != o) continue;
        int ops = 8 + 4 * IN1_D[I_IN1[p]] + 6 * OUT_D[o] + CG_BEGIN[p + 1] - CG_BEGIN[p];
        for (int c = CG_BEGIN[p]; c < CG_BEGIN[p + 1]; ++c)
            if (c == CG_BEGIN[p] || CG_I[c] != CG_I[c - 1] || CG_J[c] != CG_J[c - 1]) ++ops;
        const int stage = tc_rpc(o) * ops / 64;
        n += tc_khalves(p) * (stage > 12 ? stage : 12);
    }
    return UNIT_Y ? 16 + OUT_MUL[o] / 4 : n;
}

// Rows of the batch that this CTA forms for output O.  Large batches: the same share of the rows for every output.  Where
// a share is a few chunks, rounding it up to whole chunks for every output (and loading all weights) costs more than the
// work: the chunks of all outputs, in one list, are cut into one run per CTA (at most two outputs in most of them).
template <int O>
__device__ __forceinline__ void tc_row_range(const UvwTcParams& p, long long& lo, long long& hi) {
    if (!p.dealt) {
        lo = p.batch * blockIdx.x / gridDim.x;
        hi = p.batch * (blockIdx.x + 1) / gridDim.x;
        return;
    }
    int total = 0, before = 0;                  // (a dealt batch is small)
    sfor<0, N_OUT>([&](auto o_) {
        constexpr int o = o_;
        const int n = ((int)p.batch + tc_rpc(o) - 1) / tc_rpc(o) * tc_chunk_cost(o);
        total += n;
        if constexpr (o < O) before += n;
    });
    constexpr int COST = tc_chunk_cost(O), RPC = tc_rpc(O);
    const int from = (int)((long long)total * blockIdx.x / gridDim.x) - before;
    const int to = (int)((long long)total * (blockIdx.x + 1) / gridDim.x) - before;
    const long long a = from > 0 ? (long long)((from + COST - 1) / COST) * RPC : 0;
    const long long b = to > 0 ? (long long)((to + COST - 1) / COST) * RPC : 0;
    lo = a < p.batch ? a : p.batch;
    hi = b < p.batch ? b : p.batch;
}

constexpr int tc_d1_max(int o) {
    int m = 1;
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o && IN1_D[I_IN1[p]] > m) m = IN1_D[I_IN1[p]];
    return m;
}
constexpr int tc_d2_max(int o) {
    int m = 1;
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o && IN2_D[I_IN2[p]] > m) m = IN2_D[I_IN2[p]];
    return m;
}
// Rows of a producer step: a warp's rows of a stage (at most one of every two groups of eight) are taken in steps whose
// inputs fit 24 registers, twice (the step at work and the one on its way).
constexpr int TC_SETS = TC_PRODUCER_WARPS / 8;
constexpr int tc_rows_of_warp(int o) { return ((tc_rpc(o) + 7) / 8 + TC_SETS - 1) / TC_SETS; }
constexpr int tc_steps(int o) {
    const int per = tc_d1_max(o) + (UNIT_Y ? 0 : tc_d2_max(o)), fit = 24 / per > 0 ? 24 / per : 1;
    return (tc_rows_of_warp(o) + fit - 1) / fit;
}
// Steps of the paths into o that come before path p_end, and the path of step n.
constexpr int tc_sequence(int o, int p_end) {
    int n = 0;
    for (int p = 0; p < p_end; ++p)
        if (I_OUT[p] == o) n += tc_khalves(p) * tc_steps(o);
    return n;
}
constexpr int tc_seq_path(int o, int n) {
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o && n < tc_sequence(o, p + 1)) return p;
    return 0;
}
constexpr int tc_step_rows(int o) { return (tc_rows_of_warp(o) + tc_steps(o) - 1) / tc_steps(o); }

// ---------------------------------------------------------------------------- producers
//
// Bound by issue once the inputs' latency is hidden.  Warp w takes the rows r = w mod 8 (mod 8); the two sets of eight
// warps take alternate groups of eight rows, swapped from stage to stage so that an odd number of groups does not leave
// one set waiting.  The inputs of a step are fetched while the step before it is formed (a warp has one to three rows
// of a stage: fetched at their use they paid the L2 latency once per stage).
template <int O>
__device__ __forceinline__ bool tc_produce_output(const UvwTcParams& p, unsigned char* smem, const TcBars& bars,
                                                  long long row_lo, long long row_hi, long long& stage_it, int warp,
                                                  int lane) {
    constexpr int D3 = OUT_D[O];
    constexpr int RPC = tc_rpc(O);
    static_assert(TC_PRODUCER_WARPS % 8 == 0, "sets of eight warps");
    constexpr bool FAST = RPC % 8 == 0;
    constexpr int STEPS = tc_steps(O), R = tc_step_rows(O);
    const int w8 = warp & 7, set = warp >> 3;
    const int base = w8 * 128 + (((lane >> 2) ^ w8) << 4) + ((lane & 3) << 2);
    constexpr int SEQ = tc_sequence(O, N_INSTR);       // steps of a chunk; step n uses buffer n mod 2
    float x[2][R][tc_d1_max(O)], y[2][R][tc_d2_max(O)];
    auto first = [&](int st) { return TC_SETS == 2 ? (set + st) & 1 : set; };      // first group of eight rows in stage st
    // inputs of path P for step j of the stage with index st: half h of the chunk at b0
    auto fetch = [&](auto p_, long long b0, int h, int st, int j, auto& xv, auto& yv) {
        constexpr int P = p_;
        constexpr int a = I_IN1[P], b = I_IN2[P], D1 = IN1_D[a], D2 = IN2_D[b], MU = IN1_MUL[a];
        const int r0 = 8 * (first(st) + TC_SETS * j * R) + w8;
        const int rows = (int)(row_hi - b0 < RPC ? row_hi - b0 : RPC);
        const bool u_live = MU % 32 == 0 || h * 32 + lane < MU;
        const float* xr = p.X + (b0 + r0) * (long long)X_DIM + IN1_OFF[a] + (h * 32 + lane) * D1;
        const float* yr = p.Y + (b0 + r0) * (long long)Y_DIM + IN2_OFF[b];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const bool live = r0 + 8 * TC_SETS * i < rows;
#pragma unroll
            for (int c = 0; c < D1; ++c) xv[i][c] = live && u_live ? __ldg(xr + i * (8 * TC_SETS * X_DIM) + c) : 0.f;
            if constexpr (!UNIT_Y) {
#pragma unroll
                for (int c = 0; c < D2; ++c) yv[i][c] = live ? __ldg(yr + i * (8 * TC_SETS * Y_DIM) + c) : 0.f;
            }
        }
    };
    bool ok = true;
    if (row_lo < row_hi) fetch(IC<tc_first_path(O)>{}, row_lo, 0, (int)(stage_it & 1), 0, x[0], y[0]);
    for (long long b0 = row_lo; b0 < row_hi && ok; b0 += RPC) {
        const int rows = (int)(row_hi - b0 < RPC ? row_hi - b0 : RPC);
        sfor<0, SEQ>([&](auto n_) {
            constexpr int NN = n_, P = tc_seq_path(O, NN), KH = tc_khalves(P), W = NN - tc_sequence(O, P);
            constexpr int h = W / STEPS, j = W % STEPS;
            if (ok) {
                auto& xc = x[NN & 1];
                auto& yc = y[NN & 1];
                auto& xn = x[(NN + 1) & 1];
                auto& yn = y[(NN + 1) & 1];
                const int s = (int)(stage_it % TC_NA), odd = (int)(stage_it & 1);
                if constexpr (j + 1 < STEPS) fetch(IC<P>{}, b0, h, odd, j + 1, xn, yn);
                else if constexpr (h + 1 < KH) fetch(IC<P>{}, b0, h + 1, odd ^ 1, 0, xn, yn);
                else if constexpr (NN + 1 < SEQ) fetch(IC<tc_seq_path(O, NN + 1)>{}, b0, 0, odd ^ 1, 0, xn, yn);
                else if (b0 + RPC < row_hi) fetch(IC<tc_first_path(O)>{}, b0 + RPC, 0, odd ^ 1, 0, xn, yn);
                if (j == 0 && stage_it >= TC_NA)
                    ok = mbar_wait(bars.a_empty + s, (unsigned)((stage_it / TC_NA - 1) & 1), p.status, ERR_TC_A_EMPTY);
                if (ok) {
                    unsigned char* tile = smem + TC_OFF_A + s * TC_STAGE_BYTES;
                    const int q0 = first(odd);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const int q = q0 + TC_SETS * (j * R + i), r = 8 * q + w8;
                        if (r < rows) {
                            float t[D3];
#pragma unroll
                            for (int k = 0; k < D3; ++k) t[k] = 0.f;
                            float xy = 0.f;
                            sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto c_) {
                                constexpr int N = c_;
                                if constexpr (N == CG_BEGIN[P] || CG_I[N] != CG_I[N - 1] || CG_J[N] != CG_J[N - 1])
                                    xy = UNIT_Y ? xc[i][CG_I[N]] : xc[i][CG_I[N]] * yc[i][CG_J[N]];
                                t[CG_K[N]] = fmaf(xy, (float)CG_V[N], t[CG_K[N]]);
                            });
                            unsigned char* hq = tile + base + q * 1024;
#pragma unroll
                            for (int k = 0; k < D3; ++k) {
                                unsigned char* dst = FAST ? hq + k * (RPC / 8) * 1024 : tile + tc_swizzle(k * RPC + r, lane);
                                const float th = tf32_hi(t[k]);
                                *reinterpret_cast<float*>(dst) = th;
                                *reinterpret_cast<float*>(dst + TC_STAGE_HALF) = t[k] - th;     // exact; read as TF32 by the MMA
                            }
                        }
                    }
                    if constexpr (j + 1 == STEPS) {
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bars.a_full + s);
                        ++stage_it;
                    }
                }
            }
        });
        if constexpr (SEQ % 2 == 1) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
#pragma unroll
                for (int c = 0; c < tc_d1_max(O); ++c) x[0][i][c] = x[1][i][c];
#pragma unroll
                for (int c = 0; c < tc_d2_max(O); ++c) y[0][i][c] = y[1][i][c];
            }
        }
    }
    return ok;
}

// ---------------------------------------------------------------------------- MMA issuer (one warp, in step)
template <int O>
__device__ __forceinline__ bool tc_mma_output(const UvwTcParams& p, unsigned char* smem, const TcBars& bars,
                                              long long row_lo, long long row_hi, long long& stage_it, long long& acc_it,
                                              int& w_use, unsigned tmem_base, unsigned leader, int lane) {
    constexpr int D3 = OUT_D[O];
    constexpr int RPC = tc_rpc(O);
    constexpr int MW = tc_mwp(O);
    // Issuing a tcgen05.mma costs about 90 cycles whatever its size, so hi.hi and hi.lo go out as one MMA: the
    // lo tile of the weights follows the hi tile in shared memory, and a B descriptor over 2 MW rows covers
    // both.  The accumulator tile is then [hi.hi + lo.hi | hi.lo], summed by the epilogue.
    constexpr bool WIDE = tc_wide(O);
    constexpr int ACC_COLS = TC_ACC_COLS;
    constexpr int NACC = TC_NACC;
    constexpr unsigned IDESC = tc_instr_desc(MW), IDESC_WIDE = tc_instr_desc(2 * MW);
    constexpr int BLOCK = tc_block_bytes(O);
    if (row_lo >= row_hi) return true;
    // the weights of the previous output must not be overwritten while tensor cores still read them
    if (w_use > 0) {
        tc_commit_if(leader, bars.w_free);
        if (!warp_wait(true, bars.w_free, (unsigned)((w_use - 1) & 1), p.status, ERR_TC_W)) return false;
    }
    if (lane == 0) {
        mbar_arrive_expect_tx(bars.w_full, (unsigned)tc_w_bytes(O));
        const unsigned char* src = reinterpret_cast<const unsigned char*>(p.Wpacked) + tc_w_offset(O);
        constexpr int TOTAL = tc_w_bytes(O);
        for (int off = 0; off < TOTAL; off += 32768) {
            const int n = TOTAL - off < 32768 ? TOTAL - off : 32768;
            bulk_g2s(smem + TC_OFF_W + off, src + off, (unsigned)n, bars.w_full);
        }
    }
    __syncwarp();
    if (!warp_wait(true, bars.w_full, (unsigned)(w_use & 1), p.status, ERR_TC_W)) return false;
    ++w_use;
    const unsigned long long w_desc0 = tc_smem_desc(smem_u32(smem + TC_OFF_W));
    const unsigned long long a_desc0 = tc_smem_desc(smem_u32(smem + TC_OFF_A));
    bool ok = true, ready = false;          // ready: the next stage was seen to be full
    for (long long b0 = row_lo; b0 < row_hi && ok; b0 += RPC) {
        const int t = (int)(acc_it % NACC);
        const long long acc_use = acc_it / NACC;
        if (acc_use > 0) ok = warp_wait(ok, bars.acc_empty + t, (unsigned)((acc_use - 1) & 1), p.status, ERR_TC_ACC_EMPTY);
        if (!ok) break;
        tc_fence_after();
        const unsigned tmem_d = tmem_base + (unsigned)(t * ACC_COLS);
        unsigned accumulate = 0;
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            if constexpr (I_OUT[P] == O) {
                for (int h = 0; h < tc_khalves(P) && ok; ++h) {
                    const int s = (int)(stage_it % TC_NA);
                    const long long use = stage_it / TC_NA;
                    const bool prof = p.prof && blockIdx.x == 0 && lane == 0;
                    const long long t0 = prof ? clock64() : 0;
                    if (!ready) ok = warp_wait(ok, bars.a_full + s, (unsigned)(use & 1), p.status, ERR_TC_A_FULL);
                    const long long t1 = prof ? clock64() : 0;
                    if (ok) {
                        tc_fence_after();
                        // descriptors differ from the base ones only in the start-address field (16-byte units):
                        // one add per operand instead of rebuilding them (the issuing thread is latency bound)
                        const unsigned long long da_hi = a_desc0 + (unsigned long long)((s * TC_STAGE_BYTES) >> 4);
                        const unsigned long long da_lo = da_hi + (TC_STAGE_HALF >> 4);
                        const unsigned long long db_hi = w_desc0 + (unsigned long long)(((tc_blocks_before(O, P) + h) * 2 * BLOCK) >> 4);
                        const unsigned long long db_lo = db_hi + (BLOCK >> 4);
                        ready = mbar_test(bars.a_full + (stage_it + 1) % TC_NA, (unsigned)((stage_it + 1) / TC_NA & 1));
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            if constexpr (WIDE) {
                                tc_mma_if(leader, tmem_d, da_hi + 2 * kk, db_hi + 2 * kk, IDESC_WIDE, accumulate);
                            } else {
                                tc_mma_if(leader, tmem_d, da_hi + 2 * kk, db_hi + 2 * kk, IDESC, accumulate);
                                tc_mma_if(leader, tmem_d, da_hi + 2 * kk, db_lo + 2 * kk, IDESC, 1);
                            }
                            accumulate = 1;
                            tc_mma_if(leader, tmem_d, da_lo + 2 * kk, db_hi + 2 * kk, IDESC, 1);
                        }
                        tc_commit_if(leader, bars.a_empty + s);   // the stage may be refilled once these MMAs have read it
                        if (prof) {
                            atomicAdd(p.prof + 8, (unsigned long long)(t1 - t0));             // wait for operands
                            atomicAdd(p.prof + 9, (unsigned long long)(clock64() - t1));      // issue
                        }
                        ready = __all_sync(0xffffffffu, ready);
                    }
                    ++stage_it;
                }
            }
        });
        if (ok) tc_commit_if(leader, bars.acc_full + t);
        ++acc_it;
    }
    return ok;
}

// ---------------------------------------------------------------------------- epilogue warps
// AND-reduction of a flag over the warps of an epilogue group (hardware barrier 1 + group).
__device__ __forceinline__ bool tc_epilogue_all(bool ok, int group) {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "bar.red.and.pred p, %3, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"((unsigned)ok), "n"(TC_EPILOGUE_WARPS * 32), "r"(1 + group)
        : "memory");
    return r != 0;
}

template <int O>
__device__ __forceinline__ bool tc_epilogue_output(const UvwTcParams& p, unsigned char* smem, const TcBars& bars,
                                                   long long row_lo, long long row_hi, long long& acc_it,
                                                   unsigned tmem_base, int ewarp, int lane, int group) {
    constexpr int D3 = OUT_D[O];
    constexpr int RPC = tc_rpc(O);
    constexpr int MW = OUT_MUL[O], MWP = tc_mwp(O);
    constexpr bool WIDE = tc_wide(O);
    constexpr int ACC_COLS = TC_ACC_COLS;
    constexpr int NACC = TC_NACC;
    float* stg = reinterpret_cast<float*>(smem + TC_OFF_STG + group * TC_STG_BYTES);
    const int et = ewarp * 32 + lane;
    const bool z_aligned = (reinterpret_cast<unsigned long long>(p.Z) & 15) == 0;
    bool ok = true;
    for (long long b0 = row_lo; b0 < row_hi && ok; b0 += RPC) {
        const int rows = (int)(row_hi - b0 < RPC ? row_hi - b0 : RPC);
        const int t = (int)(acc_it % NACC);
        const long long use = acc_it / NACC;
        const bool prof = p.prof && blockIdx.x == 0 && et == 0;
        const long long t0 = prof ? clock64() : 0;
        ok = mbar_wait(bars.acc_full + t, (unsigned)(use & 1), p.status, ERR_TC_ACC_FULL);
        if (prof) atomicAdd(p.prof + 16, (unsigned long long)(clock64() - t0));
        const long long t1 = prof ? clock64() : 0;
        // the four warps must agree before anyone touches the staging buffer or skips a barrier
        ok = tc_epilogue_all(ok, group);
        if (!ok) break;
        tc_fence_after();
        // (ewarp is the warp's TMEM lane quarter) accumulator row m = 32 * ewarp + lane holds (row m % RPC, component m / RPC) for all w
        const unsigned taddr = tmem_base + ((unsigned)(ewarp * 32) << 16) + (unsigned)(t * ACC_COLS);
        constexpr int BLOCKS = (MWP + TC_BLOCK_COLS - 1) / TC_BLOCK_COLS, NT = TC_EPILOGUE_WARPS * 32;
        const int first = (group + (int)(acc_it % TC_EPI_GROUPS)) % TC_EPI_GROUPS;
        bool drained = BLOCKS <= first;             // the group has no block of this tile
        if (drained && et == 0) mbar_arrive(bars.acc_empty + t);
        auto block = [&](auto cols_, auto live_, int B) {
            constexpr int COLS = cols_, LIVE = live_;
            const int C0 = B * TC_BLOCK_COLS;
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16) {
                unsigned v[16], v2[16];
                tc_load16(taddr + (unsigned)(C0 + c0), v);
                if constexpr (WIDE) tc_load16(taddr + (unsigned)(MWP + C0 + c0), v2);   // the hi.lo half of the tile
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    float val = __uint_as_float(v[c]);
                    if constexpr (WIDE) val += __uint_as_float(v2[c]);
                    stg[(ewarp * 32 + lane) * TC_STG_PITCH + c0 + c] = val;
                }
            }
            tc_fence_before();
            asm volatile("bar.sync %1, %0;" ::"n"(NT), "r"(1 + group) : "memory");
            if (B + TC_EPI_GROUPS >= BLOCKS && et == 0) mbar_arrive(bars.acc_empty + t);    // the group is done with the tile
            // staged rows (k * RPC + row) x w  ->  Z[row][OUT_OFF + w * D3 + k], contiguous per batch row.  A thread keeps
            // four consecutive values of a row and walks the rows: no index division and a quarter of the stores.
            constexpr int ROWLEN = LIVE * D3;
            const int off0 = OUT_OFF[O] + C0 * D3;
            constexpr bool VEC = ROWLEN % 4 == 0 && OUT_OFF[O] % 4 == 0 && Z_DIM % 4 == 0;
            if (VEC && z_aligned) {
                constexpr int TPR = (ROWLEN + 3) / 4, SIDE = TPR < NT ? NT / TPR : 1;      // threads per row, rows side by side
                if (TPR >= NT || et < SIDE * TPR) {
#pragma unroll 1
                    for (int j4 = TPR < NT ? et % TPR : et; j4 < TPR; j4 += TPR < NT ? TPR : NT) {
                        int off[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) off[i] = ((4 * j4 + i) % D3 * RPC) * TC_STG_PITCH + (4 * j4 + i) / D3;
                        float* zrow = p.Z + b0 * (long long)Z_DIM + off0 + 4 * j4;
#pragma unroll 4
                        for (int r = TPR < NT ? et / TPR : 0; r < rows; r += SIDE) {
                            const float* src = stg + r * TC_STG_PITCH;
                            *reinterpret_cast<float4*>(zrow + r * (long long)Z_DIM) = make_float4(src[off[0]], src[off[1]], src[off[2]], src[off[3]]);
                        }
                    }
                }
            } else {
                for (int e = et; e < rows * ROWLEN; e += NT) {
                    const int r = e / ROWLEN, j = e - r * ROWLEN;
                    const int w = j / D3, k = j - w * D3;
                    p.Z[(b0 + r) * (long long)Z_DIM + off0 + j] = stg[(k * RPC + r) * TC_STG_PITCH + w];
                }
            }
            asm volatile("bar.sync %1, %0;" ::"n"(NT), "r"(1 + group) : "memory");
        };
        // One body for all whole blocks: a body for each does not fit the instruction caches (W dZ of 64x(0e+1o+2e) with 0e+1o+2e, 100 000
        // rows 263 -> 246 us; twice the unrolling of the stores took it from 263 to 275).
        constexpr int WHOLE = MW / TC_BLOCK_COLS;
#pragma unroll 1
        for (int B = first; B < WHOLE; B += TC_EPI_GROUPS) block(IC<TC_BLOCK_COLS>{}, IC<TC_BLOCK_COLS>{}, B);
        if constexpr (WHOLE < BLOCKS)
            if (WHOLE % TC_EPI_GROUPS == first) block(IC<MWP - WHOLE * TC_BLOCK_COLS>{}, IC<MW - WHOLE * TC_BLOCK_COLS>{}, WHOLE);
        if (prof) {
            atomicAdd(p.prof + 17, (unsigned long long)(clock64() - t1));
            atomicAdd(p.prof + 18, 1ull);
        }
        ++acc_it;
    }
    return ok;
}

constexpr bool tc_output_has_paths(int o) {
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o) return true;
    return false;
}

// Small batches: the output irreps are dealt over the grid's y dimension (a CTA that took all of them would load their
// weights one after the other while most of the machine is idle).
__device__ __forceinline__ bool tc_mine(int o) { return gridDim.y == 1 || (int)blockIdx.y == o; }

__device__ void uvw_tc_forward(const UvwTcParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the 128-byte swizzle pattern repeats every 1024 bytes: operand tiles must start on that boundary
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const TcBars bars(smem);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    long long row_lo, row_hi;

    if (tid == 0) {
        for (int i = 0; i < TC_NA; ++i) {
            mbar_init(bars.a_full + i, TC_PRODUCER_WARPS);
            mbar_init(bars.a_empty + i, 1);
        }
        for (int i = 0; i < TC_MAX_ACC; ++i) {
            mbar_init(bars.acc_full + i, 1);
            mbar_init(bars.acc_empty + i, TC_EPI_GROUPS);
        }
        mbar_init(bars.w_full, 1);
        mbar_init(bars.w_free, 1);
        fence_mbar_init();
    }
    if (warp == TC_PRODUCER_WARPS) {   // the MMA warp owns the tensor memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(bars.tmem_slot)),
                     "n"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile unsigned*>(bars.tmem_slot), 0);

    if (warp < TC_PRODUCER_WARPS) {
        long long stage_it = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            if (!tc_mine(O)) return;
            tc_row_range<O>(p, row_lo, row_hi);
            if constexpr (tc_output_has_paths(O)) {
                if (ok) ok = tc_produce_output<O>(p, smem, bars, row_lo, row_hi, stage_it, warp, lane);
            } else {
                // an output irrep that no path writes is zero
                for (long long b = row_lo + warp; b < row_hi; b += TC_PRODUCER_WARPS)
                    for (int j = lane; j < OUT_MUL[O] * OUT_D[O]; j += 32) p.Z[b * (long long)Z_DIM + OUT_OFF[O] + j] = 0.f;
            }
        });
    } else if (warp == TC_PRODUCER_WARPS) {
        const unsigned leader = elect_lane();
        long long stage_it = 0, acc_it = 0;
        int w_use = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            if (!tc_mine(O)) return;
            tc_row_range<O>(p, row_lo, row_hi);
            if constexpr (tc_output_has_paths(O)) {
                if (ok) ok = tc_mma_output<O>(p, smem, bars, row_lo, row_hi, stage_it, acc_it, w_use, tmem_base, leader, lane);
            }
        });
        __syncwarp();
    } else {
        long long acc_it = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            if (!tc_mine(O)) return;
            tc_row_range<O>(p, row_lo, row_hi);
            if constexpr (tc_output_has_paths(O)) {
                // a warp may only read the TMEM lanes of its own quarter: 32 * (warp index mod 4)
                if (ok) ok = tc_epilogue_output<O>(p, smem, bars, row_lo, row_hi, acc_it, tmem_base, warp & 3, lane, (warp - TC_PRODUCER_WARPS - 1) / TC_EPILOGUE_WARPS);
            }
        });
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TC_PRODUCER_WARPS) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TC_TMEM_COLS) : "memory");
    }
}

}  // namespace oeq

#define OEQ_K_UVW_TC_FWD 20

extern "C" __global__ void __launch_bounds__(oeq::TC_THREADS, 1) oeq_uvw_tc_kernel(const oeq::UvwTcParams p) {
    oeq::uvw_tc_forward(p);
}

// Splits the shared weights into TF32 hi / lo parts and lays them out as the B operand of the MMA:
// per output irrep, per path into it, per 32-wide slice of u, a [mul_out x 32] K-major tile with the
// 128-byte swizzle for hi and one for lo.  Rows of u beyond the multiplicity are zero.
extern "C" __global__ void oeq_uvw_pack_weights(const float* __restrict__ W, float* __restrict__ packed) {
    using namespace oeqd;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    oeq::sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        if (blockIdx.y != P) return;
        constexpr int O = I_OUT[P], MU = IN1_MUL[I_IN1[P]], MW = OUT_MUL[O], MWP = oeq::tc_mwp(O);
        constexpr int KH = oeq::tc_khalves(P), BLOCK = oeq::tc_block_bytes(O);
        unsigned char* base = reinterpret_cast<unsigned char*>(packed) + oeq::tc_w_offset(O) +
                              oeq::tc_blocks_before(O, P) * 2 * BLOCK;
        for (int e = tid; e < KH * MWP * 32; e += nthreads) {
            const int col = e & 31, w = (e >> 5) % MWP, h = e / (32 * MWP);
            const int u = h * 32 + col;
            float v = 0.f;
            if (u < MU && w < MW) {
                if constexpr (TRANSPOSED_W) {
                    // output channels are those of several paths: the weights of path q, [its channels][MU], from row SUB_START[q] on
                    oeq::sfor<SUB_BEGIN[P], SUB_BEGIN[P + 1]>([&](auto q_) {
                        constexpr int q = q_;
                        if (w >= SUB_START[q] && w < SUB_START[q] + SUB_MUL[q])
                            v = W[SUB_WOFF[q] + oeq::weight_offset_v1(SUB_MUL[q], MU, w - SUB_START[q], u)];
                    });
                } else {
                    v = W[W_OFF[P] + oeq::weight_offset_v1(MU, MW, u, w)];
                }
            }
            const float hi = oeq::tf32_round(v), lo = oeq::tf32_round(v - hi);
            unsigned char* blk = base + h * 2 * BLOCK;
            *reinterpret_cast<float*>(blk + oeq::tc_swizzle(w, col)) = hi;
            *reinterpret_cast<float*>(blk + BLOCK + oeq::tc_swizzle(w, col)) = lo;
        }
    });
}
