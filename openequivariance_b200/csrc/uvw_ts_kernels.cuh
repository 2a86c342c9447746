// "uvw" forward pass on the 5th-generation tensor cores with the weights in tensor memory: shared FP32 weights, second
// input of multiplicity 1, at most 64 output channels per irrep.  FP32 in / FP32 out, 3xTF32.
//
//   Z[b,o,w,k] = sum_{paths p -> o} sum_u W_p[u,w] T_p[b,u,k],   T_p[b,u,k] = sum_i M_p[b,i,k] x[b,u,i],  M_p = sum_j C_p y_j
//
// The weights are the A operand: rows 0-63 of an MMA are the TF32 hi parts of 64 output channels, rows 64-127 the lo parts,
// and stay in tensor memory for as long as the CTA works on an output irrep (columns: the input channels of all its paths).
// T is the B operand, [(component, batch row) x 32 input channels] for 16 batch rows, hi tile followed by lo tile.  The four
// quarters of the accumulator, hi.hi, hi.lo, lo.hi and lo.lo, are added by the epilogue.
//   * 16 producer warps in four sets, each the builder of one slot of the stage ring: a thread has one batch row and four
//     input channels; it forms M of its row and path once per slice and applies it to its channels, reads x and writes T in
//     16-byte pieces.  Which four channels depends on the row such that neither the reads (rows of X as they are in memory) nor
//     the writes (128-byte swizzle) meet on a bank.
//   * one warp issues the MMAs.  All its lanes walk the loop and one issues: operands are then in uniform registers and an MMA
//     takes 20 cycles of issue; issued from a divergent lane it took 88, whatever its size.
//   * 4 epilogue warps add hi and lo rows and store rows of Z; the first one copies the rows of X and Y (consecutive in
//     memory: one bulk copy per tile and array).
// Every wait is bounded; on expiry the role records a code in *status and goes through the rest of its barriers without
// work, and the CTA frees its tensor memory.
// Measured against uvw_tc_kernels.cuh (weights in shared memory, which then has no room for rows of X), 64x(0e+1o+2e) with
// 0e+1o+2e, calls from a cold cache, with the packing of the weights: 100 000 rows 413 -> 272 us, 10 000 67 -> 46, 4 000 44 -> 31,
// 1 000 30 -> 23, 20 rows 33 -> 20; relative error against 64 bits 1.2e-6 -> 6.2e-7 (hi.lo has accumulators of its own).  Problems of few
// slices of input channels are slower here and keep the other kernel (uvw_ts_faster in the runtime).
// Bound by shared memory: per batch row 140 cycles of T's stores, 140 of the MMAs reading it, 80 of x and y, 72 of the epilogue
// and 54 of the input copies, and conflicts between them, of 700; the tensor pipe is busy for 37 %, issue slots for 42 %.
#pragma once
#include "oeq_common.cuh"
#include "uvw_ts_common.cuh"

namespace oeq {
using namespace oeqd;

struct UvwTsParams {
    const float* X;
    const float* Y;
    const float* W;
    float* Z;
    long long batch;
    int* status;
    int in_vec, z_vec;          // X and Y, and Z, start on a 16-byte boundary
};

constexpr int TS_ROWS = 16;                     // batch rows of a tile
constexpr int TS_STAGES = 4, TS_SET = 4;        // slots of the stage ring, producer warps of each
constexpr int TS_PW = TS_STAGES * TS_SET, TS_EW = 4;    // producer and epilogue warps
constexpr int TS_THREADS = (TS_PW + TS_EW + 1) * 32;
constexpr int ERR_TS_EMPTY = 51, ERR_TS_FULL = 52, ERR_TS_ACC_EMPTY = 53, ERR_TS_ACC_FULL = 54, ERR_TS_IN = 55, ERR_TS_IN_EMPTY = 56;

// ---- compile-time geometry
constexpr int ts_n(int o) { return TS_ROWS * OUT_D[o]; }                        // N of the MMA, of a hi or lo tile
constexpr int TS_W_COLS = 256, TS_ACC_COLS = 256, TS_BUFS = 4;  // tensor memory: weights, accumulators
constexpr int ts_bufs(int o) { return TS_ACC_COLS / (2 * ts_n(o)) < TS_BUFS ? TS_ACC_COLS / (2 * ts_n(o)) : TS_BUFS; }
// Shared memory while the CTA works on output o (1024-byte aligned base): [stages][rows of Z from hi and from lo
// weights][rows of X and Y of two to four tiles].  The inputs of a small tile are used up faster than memory answers.
constexpr int TS_X_BYTES = TS_ROWS * X_DIM * 4, TS_Y_BYTES = TS_ROWS * Y_DIM * 4, TS_IN = TS_X_BYTES + TS_Y_BYTES, TS_IN_MAX = 4;
constexpr int ts_stage(int o) { return 2 * ts_n(o) * 128; }                     // hi and lo tile, [N x 32] each
constexpr int ts_stg(int o) { return TS_ROWS * OUT_MUL[o] * OUT_D[o] * 4; }
constexpr int ts_off_stg(int o) { return TS_STAGES * ts_stage(o); }
constexpr int ts_off_in(int o) { return ts_off_stg(o) + 2 * ts_stg(o); }
constexpr int ts_data() {
    int m = 0;
    for (int o = 0; o < N_OUT; ++o) m = ts_slices(o) && ts_off_in(o) + 2 * TS_IN > m ? ts_off_in(o) + 2 * TS_IN : m;
    return m;
}
constexpr int ts_ins(int o) { return (ts_data() - ts_off_in(o)) / TS_IN < TS_IN_MAX ? (ts_data() - ts_off_in(o)) / TS_IN : TS_IN_MAX; }
// An output of fewer slices than there are sets of producers: a set without a slice in a tile reads its inputs all the same (and waits
// for each, or it would miss a phase), and the tile's accumulator says nothing of that set.  Its input buffers have barriers of
// their own.  With more slices every set has a part in every accumulator.
constexpr bool ts_idle_sets(int o) { return ts_slices(o) < TS_STAGES; }
constexpr int TS_BARS = 2 * TS_STAGES + 2 * TS_BUFS + 2 * TS_IN_MAX;        // of each output: no phase outlives an output
constexpr int TS_OFF_BAR = ts_data();
constexpr int TS_SMEM = TS_OFF_BAR + N_OUT * TS_BARS * 8 + 16 + 1024;           // + alignment slack

struct TsBars {
    unsigned long long *full, *empty, *acc_full, *acc_empty, *in_full, *in_empty;
    __device__ TsBars(unsigned char* smem, int o) {
        full = reinterpret_cast<unsigned long long*>(smem + TS_OFF_BAR) + o * TS_BARS;
        empty = full + TS_STAGES; acc_full = empty + TS_STAGES; acc_empty = acc_full + TS_BUFS;
        in_full = acc_empty + TS_BUFS; in_empty = in_full + TS_IN_MAX;
    }
};

// Time of a tile.  Measured for 1 / 2 / 4 / 8 slices, in units of 6 cycles: 216 / 262 / 308 / 400 of one component, 324 / 370 / 450 / 636
// of three, 384 / 494 / 632 / 882 of five, 462 / 614 of seven (one and two slices); 330 for six of one.  Mostly the drain, which takes as long for one
// slice as for eight: with a cost in proportion to the slices an output of one slice got too few CTAs (64x(0e+1o+2e) + 32x0o with
// 0e+1o+2e to 64x(1o+2e) + 16x0o, 100 000 rows: 1 002 us, now 288; 64x(0e+1o+2e) with 0e+1o 227 and 204).
constexpr int ts_cost(int o) { return ts_slices(o) ? 140 + 40 * OUT_D[o] + ts_slices(o) * (13 + 11 * OUT_D[o]) : 0; }

// MMA with the A operand in tensor memory, issued by the lane whose `leader` is set; every lane of the warp comes here.
__device__ __forceinline__ void tc_mma_ts(unsigned leader, unsigned tmem_d, unsigned tmem_a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(leader)
        : "memory");
}
// ---------------------------------------------------------------------------- producers
template <int O>
__device__ __forceinline__ void ts_produce(const UvwTsParams& p, unsigned char* smem, const TsBars& bars, int tile_lo, int tile_hi,
                                           bool& ok, int warp, int lane) {
    constexpr int INS = ts_ins(O);
    const int set = warp / TS_SET, r = lane & 15, r8 = r & 7;
    // Four channels of a slice: the threads of row r take them in the order j ^ L(r), where L is a product with x in GF(8): L
    // and L + 1 are invertible, so eight rows read eight places of a row (an odd number of pieces apart) and write eight pieces.
    const int group = ((lane >> 4) + 2 * (warp % TS_SET)) ^ ((r8 << 1 & 7) ^ (r8 & 4 ? 3 : 0));
    unsigned char* dst = smem + set * ts_stage(O) + (r >> 3) * 1024 + r8 * 128 + ((group ^ r8) << 4);
    int stage_it = 0, b = 0;
    unsigned phase = 0;             // of the input buffers
    for (int tile = tile_lo; tile < tile_hi; ++tile) {
        unsigned char* in = smem + ts_off_in(O) + b * TS_IN;
        if (p.in_vec) {
            ok = warp_wait(ok, bars.in_full + b, phase, p.status, ERR_TS_IN);
        } else {
            const long long row0 = (long long)tile * TS_ROWS;
            const int rows = (int)(p.batch - row0 < TS_ROWS ? p.batch - row0 : TS_ROWS), tid = warp * 32 + lane;
            for (int i = tid; i < rows * X_DIM; i += TS_PW * 32) reinterpret_cast<float*>(in)[i] = __ldg(p.X + row0 * X_DIM + i);
            for (int i = tid; i < rows * Y_DIM; i += TS_PW * 32) reinterpret_cast<float*>(in + TS_X_BYTES)[i] = __ldg(p.Y + row0 * Y_DIM + i);
            group_sync(1, TS_PW * 32);      // (the rows that were in this buffer have been read: the barrier of the tile between)
        }
        const float* x_row = reinterpret_cast<const float*>(in) + r * X_DIM;
        const float* y_row = reinterpret_cast<const float*>(in + TS_X_BYTES) + r * Y_DIM;
        float y_regs[Y_DIM <= 16 ? Y_DIM : 1] = {};     // (shared memory's bandwidth bounds the kernel)
        if constexpr (Y_DIM <= 16) {
#pragma unroll
            for (int j = 0; j < Y_DIM; ++j) y_regs[j] = y_row[j];
        }
        auto y = [&](int j) { return Y_DIM <= 16 ? y_regs[Y_DIM <= 16 ? j : 0] : y_row[j]; };
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            if constexpr (I_OUT[P] == O) {
                constexpr int A = I_IN1[P], D1 = IN1_D[A], MU = IN1_MUL[A], KH = ts_halves(P);
#pragma unroll 1
                for (int h = (set - stage_it) & (TS_STAGES - 1); h < KH; h += TS_STAGES) {
                    const int use = (stage_it + h) / TS_STAGES;
                    if (use > 0) ok = warp_wait(ok, bars.empty + set, (unsigned)(use - 1) & 1, p.status, ERR_TS_EMPTY);
                    if (ok) {
                        float x[4 * D1];
                        const int u0 = 32 * h + 4 * group;
#pragma unroll
                        for (int c = 0; c < D1; ++c) {
                            const float4 q = MU % 32 == 0 || u0 < MU ? *reinterpret_cast<const float4*>(x_row + IN1_OFF[A] + u0 * D1 + 4 * c)
                                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
                            x[4 * c] = q.x; x[4 * c + 1] = q.y; x[4 * c + 2] = q.z; x[4 * c + 3] = q.w;
                        }
                        ts_form<P>(x, y, [&](auto k_, float4 hi, float4 lo) {
                            constexpr int K = k_;
                            *reinterpret_cast<float4*>(dst + K * 2048) = hi;
                            *reinterpret_cast<float4*>(dst + K * 2048 + ts_n(O) * 128) = lo;
                        });
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bars.full + set);
                    }
                }
                stage_it += KH;
            }
        });
        if constexpr (ts_idle_sets(O)) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bars.in_empty + b);
        }
        if (++b == INS) {
            b = 0;
            phase ^= 1;
        }
    }
}

// ---------------------------------------------------------------------------- MMA issuer (one warp)
// What it does per slice is on the critical path, since slices are taken in order: the barrier of the next slice is looked at
// before the MMAs of this one go out.  T's hi and lo tiles lie one after the other and are one operand: beside producers
// that keep shared memory busy every MMA takes about 40 cycles more than its columns do.
template <int O>
__device__ __forceinline__ void ts_mma(const UvwTsParams& p, unsigned char* smem, const TsBars& bars, int tile_lo, int tile_hi, bool& ok,
                                       unsigned tmem_base, unsigned leader) {
    constexpr int N = ts_n(O), BUFS = ts_bufs(O), SLICES = ts_slices(O);
    constexpr unsigned IDESC = tc_instr_desc(2 * N);
    static_assert((TS_STAGES & (TS_STAGES - 1)) == 0, "slot and phase of a slice are bits of its number");
    const unsigned long long desc0 = tc_smem_desc(smem_u32(smem));
    int t = 0, rounds = 0, it = 0;
    bool ready = false;                     // slice `it` was seen to be full
    for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
        if (rounds > 0) ok = warp_wait(ok, bars.acc_empty + t, (unsigned)(rounds - 1) & 1, p.status, ERR_TS_ACC_EMPTY);
        const unsigned tmem_d = tmem_base + TS_W_COLS + (unsigned)(t * 2 * N);
#pragma unroll 1
        for (int c = 0; c < SLICES && ok; ++c, ++it) {
            const int s = it % TS_STAGES;
            if (!ready) ok = warp_wait(ok, bars.full + s, (unsigned)(it / TS_STAGES) & 1, p.status, ERR_TS_FULL);
            if (!ok) break;
            tc_fence_after();
            ready = mbar_test(bars.full + (it + 1) % TS_STAGES, (unsigned)((it + 1) / TS_STAGES) & 1);
            const unsigned long long b = desc0 + (unsigned long long)((s * ts_stage(O)) >> 4);
            const unsigned tmem_a = tmem_base + (unsigned)(32 * c);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) tc_mma_ts(leader, tmem_d, tmem_a + (unsigned)(8 * kk), b + 2 * kk, IDESC, c > 0 || kk > 0);
            tc_commit_if(leader, bars.empty + s);
            ready = __all_sync(0xffffffffu, ready);
        }
        if (ok) tc_commit_if(leader, bars.acc_full + t);
        if (++t == BUFS) {
            t = 0;
            ++rounds;
        }
    }
}

// ---------------------------------------------------------------------------- weights, epilogue warps
// Weights of output O: TMEM row l is output channel l mod 64, hi parts in rows 0-63, lo parts in 64-127.  A warp writes the
// rows of its quarter (warp mod 4), slices turn, turn + turns, ... of 32 input channels.
template <int O>
__device__ __forceinline__ void ts_load_weights(const UvwTsParams& p, unsigned tmem_base, int quarter, int lane, int turn, int turns) {
    constexpr int MW = OUT_MUL[O];
    const int row = quarter * 32 + lane, w = row & 63;
    const bool lo = row >= 64;
    const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16);
    sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        if constexpr (I_OUT[P] == O) {
            constexpr int MU = IN1_MUL[I_IN1[P]];
            sfor<0, ts_halves(P)>([&](auto h_) {
                constexpr int H = h_, C = ts_column(P) / 32 + H, ULEN = MU - 32 * H < 32 ? MU - 32 * H : 32;
                if (C % turns == turn) {
                    // 32-wide chunks [input channel][output channel]
                    const int wc = w >> 5, wlen = MW - 32 * wc < 32 ? MW - 32 * wc : 32;
                    const float* src = p.W + W_OFF[P] + 32 * H * MW + ULEN * 32 * wc + (w & 31);
                    float q[32];
#pragma unroll
                    for (int c = 0; c < 32; ++c) q[c] = c < ULEN && w < MW ? __ldg(src + c * wlen) : 0.f;
#pragma unroll
                    for (int c0 = 0; c0 < 32; c0 += 16) {
                        unsigned v[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const float hi = tf32_hi(q[c0 + c]);
                            v[c] = __float_as_uint(lo ? tf32_hi(q[c0 + c] - hi) : hi);
                        }
                        tc_store16(taddr + (unsigned)(32 * C + c0), v);
                    }
                }
            });
        }
    });
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    tc_fence_before();
}

// (one warp) rows of X and Y of a tile into input buffer b
template <int O>
__device__ __forceinline__ void ts_copy_rows(const UvwTsParams& p, unsigned char* smem, const TsBars& bars, int tile, int b, unsigned leader, int lane) {
    unsigned char* in = smem + ts_off_in(O) + b * TS_IN;
    const long long row0 = (long long)tile * TS_ROWS;
    const int rows = (int)(p.batch - row0 < TS_ROWS ? p.batch - row0 : TS_ROWS);
    const bool all = rows == TS_ROWS;
    if (!all) {                             // (a part of the rows of Y need not be whole 16-byte pieces)
        for (int i = lane; i < rows * Y_DIM; i += 32) reinterpret_cast<float*>(in + TS_X_BYTES)[i] = __ldg(p.Y + row0 * Y_DIM + i);
        __syncwarp();
    }
    expect_tx_if(leader, bars.in_full + b, (unsigned)(rows * X_DIM * 4 + (all ? TS_Y_BYTES : 0)));
    bulk_g2s_if(leader, in, p.X + row0 * X_DIM, (unsigned)(rows * X_DIM * 4), bars.in_full + b);
    if (all) bulk_g2s_if(leader, in + TS_X_BYTES, p.Y + row0 * Y_DIM, TS_Y_BYTES, bars.in_full + b);
}

// The first of its warps copies the inputs: a tile's accumulator is complete, so its rows of X and Y have been read by the sets that had
// a slice of it; ts_idle_sets.
template <int O>
__device__ __forceinline__ void ts_epilogue(const UvwTsParams& p, unsigned char* smem, const TsBars& bars, int tile_lo, int tile_hi,
                                            bool& ok, unsigned tmem_base, unsigned leader, int ewarp, int lane) {
    constexpr int INS = ts_ins(O), D3 = OUT_D[O], MW = OUT_MUL[O], N = ts_n(O), BUFS = ts_bufs(O), ROWLEN = MW * D3, NT = TS_EW * 32;
    const int et = ewarp * 32 + lane, w = et & 63;
    float* hi_rows = reinterpret_cast<float*>(smem + ts_off_stg(O));
    const float* lo_rows = hi_rows + ts_stg(O) / 4;
    float* stg = hi_rows + (et >> 6) * (ts_stg(O) / 4) + w * D3;
    const bool copies = ewarp == 0 && p.in_vec;
    if (copies)
        for (int i = 0; i < INS && tile_lo + i < tile_hi; ++i) ts_copy_rows<O>(p, smem, bars, tile_lo + i, i, leader, lane);
    int t = 0, b = 0;
    unsigned phase = 0, in_phase = 0;
    for (int tile = tile_lo; tile < tile_hi; ++tile) {
        const long long row0 = (long long)tile * TS_ROWS;
        const int rows = (int)(p.batch - row0 < TS_ROWS ? p.batch - row0 : TS_ROWS);
        ok = warp_wait(ok, bars.acc_full + t, phase, p.status, ERR_TS_ACC_FULL);
        if (copies && tile + INS < tile_hi) {
            if constexpr (ts_idle_sets(O)) ok = warp_wait(ok, bars.in_empty + b, in_phase, p.status, ERR_TS_IN_EMPTY);
            if (ok) ts_copy_rows<O>(p, smem, bars, tile + INS, b, leader, lane);
        }
        if (++b == INS) {
            b = 0;
            in_phase ^= 1;
        }
        if (ok) {
            tc_fence_after();
            // column n of either half of the tile: component n / 16 of batch row n mod 16
            const unsigned taddr = tmem_base + ((unsigned)(ewarp * 32) << 16) + (unsigned)(TS_W_COLS + t * 2 * N);
#pragma unroll
            for (int k = 0; k < D3; ++k) {
                unsigned v[2][16];
                tc_load16(taddr + (unsigned)(16 * k), v[0]);
                tc_load16(taddr + (unsigned)(N + 16 * k), v[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (w < MW) {
#pragma unroll
                    for (int r = 0; r < 16; ++r) stg[r * ROWLEN + k] = __uint_as_float(v[0][r]) + __uint_as_float(v[1][r]);
                }
            }
            tc_fence_before();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.acc_empty + t);
        if (++t == BUFS) {
            t = 0;
            phase ^= 1;
        }
        group_sync(2, NT);
        if (ok) {
            constexpr bool VEC = ROWLEN % 4 == 0 && OUT_OFF[O] % 4 == 0 && Z_DIM % 4 == 0;
            float* z0 = p.Z + row0 * Z_DIM + OUT_OFF[O];
            if (VEC && p.z_vec) {
#pragma unroll 4
                for (int i = et; i < rows * (ROWLEN / 4); i += NT) {
                    const int r = i / (ROWLEN / 4), c = i - r * (ROWLEN / 4);
                    const float4 a = *reinterpret_cast<const float4*>(hi_rows + 4 * i), b = *reinterpret_cast<const float4*>(lo_rows + 4 * i);
                    *reinterpret_cast<float4*>(z0 + r * (long long)Z_DIM + 4 * c) = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
                }
            } else {
                for (int i = et; i < rows * ROWLEN; i += NT) {
                    const int r = i / ROWLEN, c = i - r * ROWLEN;
                    z0[r * (long long)Z_DIM + c] = hi_rows[i] + lo_rows[i];
                }
            }
        }
        group_sync(2, NT);
    }
}

__device__ void uvw_ts_forward(const UvwTsParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the 128-byte swizzle pattern repeats every 1024 bytes: operand tiles must start on that boundary
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + TS_OFF_BAR + N_OUT * TS_BARS * 8);
    if (tid == 0) {
        for (int o = 0; o < N_OUT; ++o) {
            const TsBars bars(smem, o);
            for (int i = 0; i < TS_STAGES; ++i) {
                mbar_init(bars.full + i, TS_SET);
                mbar_init(bars.empty + i, 1);
            }
            for (int i = 0; i < TS_BUFS; ++i) {
                mbar_init(bars.acc_full + i, 1);
                mbar_init(bars.acc_empty + i, TS_EW);
            }
            for (int i = 0; i < TS_IN_MAX; ++i) {
                mbar_init(bars.in_full + i, 1);
                mbar_init(bars.in_empty + i, TS_PW);
            }
        }
        fence_mbar_init();
    }
    if (warp == TS_PW + TS_EW) {        // the MMA warp owns the tensor memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "n"(TS_W_COLS + TS_ACC_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile unsigned*>(tmem_slot), 0);
    const unsigned leader = elect_lane();
    bool ok = true;
    sfor<0, N_OUT>([&](auto o_) {
        constexpr int O = o_;
        if constexpr (ts_slices(O) > 0) {
            int lo, hi;
            ts_deal<O, TS_ROWS, ts_cost>(p.batch, blockIdx.x, gridDim.x, gridDim.x, lo, hi);
            if (lo < hi) {
                const TsBars bars(smem, O);
                // (the output before is complete: its shared and tensor memory are free)
                if (warp < TS_PW + TS_EW) ts_load_weights<O>(p, tmem_base, warp & 3, lane, warp >> 2, (TS_PW + TS_EW) / 4);
                tc_fence_before();
                __syncthreads();
                tc_fence_after();
                if (warp < TS_PW) ts_produce<O>(p, smem, bars, lo, hi, ok, warp, lane);
                else if (warp < TS_PW + TS_EW) ts_epilogue<O>(p, smem, bars, lo, hi, ok, tmem_base, leader, warp - TS_PW, lane);
                else ts_mma<O>(p, smem, bars, lo, hi, ok, tmem_base, leader);
                fence_async_smem();         // (what was a stage may be the destination of bulk copies next)
                tc_fence_before();
                ok = __syncthreads_and(ok);
                tc_fence_after();
            }
        } else if (warp < TS_PW) {
            // an output irrep that no path writes is zero
            const long long lo = p.batch * blockIdx.x / gridDim.x, hi = p.batch * (blockIdx.x + 1) / gridDim.x;
            for (long long b = lo + warp; b < hi; b += TS_PW)
                for (int j = lane; j < OUT_MUL[O] * OUT_D[O]; j += 32) p.Z[b * (long long)Z_DIM + OUT_OFF[O] + j] = 0.f;
        }
    });
    tc_fence_before();
    __syncthreads();
    if (warp == TS_PW + TS_EW)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TS_W_COLS + TS_ACC_COLS) : "memory");
}

}  // namespace oeq

#define OEQ_K_UVW_TS_FWD 22

extern "C" __global__ void __launch_bounds__(oeq::TS_THREADS, 1) oeq_uvw_ts_kernel(const oeq::UvwTsParams p) { oeq::uvw_ts_forward(p); }
