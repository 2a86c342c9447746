// Weight gradient of the "uvw" product on the 5th-generation tensor cores from rows formed a batch row per lane: shared FP32
// weights, second input of multiplicity 1, at most 64 output channels per irrep.  FP32 in / FP32 out, 3xTF32.
//
//   dW_p[u,w] = sum_{b,k} T_p[b,u,k] dZ[b,o,w,k],   T_p[b,u,k] = sum_i M_p[b,i,k] x[b,u,i],  M_p = sum_j C_p y_j
//
// The sum runs over batch rows and components, so both operands have the channels along their rows: T [(k, b) x u] and
// dZ [(k, b) x w], "MN-major" tiles of 32 channels by 8 batch rows per component (128-byte rows, 32-byte atoms swizzled over four
// rows).  That is the order in which a thread with one batch row forms them, as in uvw_ts_kernels.cuh: its matrix M serves four
// channels, and rows of X and dZ come as bulk copies.  An MMA tile has the channels of four slices of 32 (128 rows); hi.hi
// and hi.lo are one MMA over dZ's hi channels followed by its lo channels, lo.hi a second one into hi.hi's columns.  The sums of all the CTA's
// rows stay in tensor memory; per CTA and output irrep they go to scratch and are added in a fixed order.
//   * 16 warps form T, in two sets with a slot of the ring each, and drain tensor memory; 4 warps split dZ and copy the
//     inputs; one warp, in step, issues the MMAs.
// uvw_tc_bwd_kernels.cuh (wider outputs) forms K-major tiles with a channel per thread: M has to be applied to every channel's
// products there, and rows of X and dZ are read from memory with a stride of 2l+1 values.
// Every wait is bounded; on expiry the role records a code in *status and goes through the rest of its barriers without
// work, and the CTA frees its tensor memory.
// Measured, 64x(0e+1o+2e) with 0e+1o+2e, calls with the sum over CTAs, uvw_tc_bwd_kernels.cuh / this kernel: 100 000 rows 517 / 380 us, 10 000
// 99 / 73, 1 000 65 / 40, but 500 rows 24 / 38 and 20 rows 20 / 32, which the wider kernel therefore takes, as it does many rows of scalar outputs
// (uvw_dw_choice in the runtime).  At 30 000 rows issue slots are busy for 53 %, the load and store unit for 41 %, the tensor pipe for
// 20 %; waits at barriers are the rest.
#pragma once
#include "oeq_common.cuh"
#include "uvw_ts_common.cuh"

namespace oeq {
using namespace oeqd;

struct UvwTsDwParams {
    const float* X;
    const float* Y;
    const float* dZ;
    float* ws;                  // [most][W_NUMEL] partial weight gradients: CTA n of those of an output writes that output's part of [n]
    long long batch;
    int* status;
    int in_vec;                 // X, Y and dZ start on a 16-byte boundary
    int most;                   // CTAs of an output at most
};

constexpr int TG_ROWS = 8;                      // batch rows of a tile: the K of an MMA
constexpr int TG_SETS = 2, TG_SET = 8;          // sets of warps that form T
constexpr int TG_ROOM = 222 * 1024;              // shared memory for operands and inputs, where it is of use
constexpr int TG_PW = TG_SETS * TG_SET, TG_BW = 4, TG_THREADS = (TG_PW + TG_BW + 1) * 32;
// Runs of tiles that the MMAs sum in one accumulator: an MMA adds to it less exactly than a rounded sum, and the error grows with the
// length of a chain.  After a run the accumulators are added to sums, in tensor memory too, while the MMAs go on in others.  The
// boundaries are those of the row ranges that the CTAs of uvw_tc_bwd_kernels.cuh have, so that the two kernels round much alike; ranges of
// more than TG_CHAIN tiles are cut into equal runs, so that the error does not go on growing.  64x(0e+1o+2e) with 0e+1o+2e, relative
// errors at 5 000 / 20 000 / 100 000 / 400 000 rows: 6.5e-7 / 2.4e-6 / 6.2e-6 / 8.6e-6, with whole ranges 6.5e-7 / 2.4e-6 / 1.2e-5 / 4.7e-5.
// (Runs of 40 / components tiles, with lo.hi beside hi.lo, cost the same and are 7.8e-7 off at 100 000 rows, but then 1.3e-5 from
// the wider kernel.)
constexpr unsigned TG_CHAIN = 64;
struct TgSegments {
    int i, next;                                // the next boundary
    static __device__ unsigned tiles(long long batch) { return (unsigned)((batch + TG_ROWS - 1) / TG_ROWS); }
    static __device__ unsigned parts(long long batch) {         // each range in equal runs
        const unsigned t = tiles(batch), ranges = min((t + 3) / 4, gridDim.x);
        return ranges * ((t + ranges * TG_CHAIN - 1) / (ranges * TG_CHAIN));
    }
    __device__ TgSegments(long long batch, int tile_lo) : i((unsigned)tile_lo / (tiles(batch) / parts(batch) + 1)) {
        do advance(batch); while (next <= tile_lo);
    }
    __device__ void advance(long long batch) {  // boundary i of all: tiles * i / parts
        const unsigned t = tiles(batch), p = parts(batch);
        ++i;
        next = (int)(i * (t / p) + (unsigned)((unsigned long long)i * (t % p) / p));
    }
    __device__ int count(long long batch, int tile_hi) {        // segments of the CTA's run
        int n = 1;
        for (; next < tile_hi; ++n) advance(batch);
        return n;
    }
};
constexpr int TG_BUFS = 3, TG_COLS = 512;       // accumulators of 128 columns, then sums of 64 for each MMA tile
constexpr int TG_B = 2, TG_IN_MAX = 4;          // slots of dZ, buffers of inputs (two to four, as they fit)
constexpr int ERR_TG_EMPTY = 61, ERR_TG_FULL = 62, ERR_TG_IN = 63, ERR_TG_IN_EMPTY = 64, ERR_TG_ACC_FULL = 65, ERR_TG_B_EMPTY = 66, ERR_TG_B_FULL = 67, ERR_TG_ACC_EMPTY = 68;

constexpr int tg_mtiles(int o) { return (ts_slices(o) + 3) / 4; }
constexpr int tg_block(int o) { return 1024 * OUT_D[o]; }                       // 32 channels of all components
constexpr int tg_a_slot(int o) { return 8 * tg_block(o); }                      // hi of four slices, lo
constexpr int tg_b_slot(int o) { return (2 * OUT_MUL[o] + 31) / 32 * tg_block(o); }      // channels hi, then lo
// Inputs of a tile: rows of X, of the output irrep's part of dZ, of Y.
constexpr int TG_X_BYTES = TG_ROWS * X_DIM * 4, TG_Y_BYTES = TG_ROWS * Y_DIM * 4;
constexpr int tg_z_len(int o) { return OUT_MUL[o] * OUT_D[o]; }
constexpr int tg_y_at(int o) { return TG_X_BYTES + TG_ROWS * tg_z_len(o) * 4; }
constexpr int tg_in(int o) { return tg_y_at(o) + TG_Y_BYTES; }
// shared memory while the CTA works on output o (1024-byte aligned base): [slots of T][slots of dZ][inputs]; [barriers]
constexpr int tg_off_b(int o) { return TG_SETS * tg_a_slot(o); }
constexpr int tg_off_in(int o) { return tg_off_b(o) + TG_B * tg_b_slot(o); }
constexpr int tg_data() {
    int m = 0;
    for (int o = 0; o < N_OUT; ++o)
        if (ts_slices(o) && tg_off_in(o) + 2 * tg_in(o) > m) m = tg_off_in(o) + 2 * tg_in(o);
    return m > TG_ROOM ? m : TG_ROOM;
}
constexpr int tg_ins(int o) { return (tg_data() - tg_off_in(o)) / tg_in(o) < TG_IN_MAX ? (tg_data() - tg_off_in(o)) / tg_in(o) : TG_IN_MAX; }
constexpr int TG_OFF_BAR = tg_data();
constexpr int TG_BARS = 2 * TG_SETS + 2 * TG_B + 2 * TG_IN_MAX + 2 * TG_BUFS;             // of each output: no phase outlives an output
constexpr int TG_SMEM = TG_OFF_BAR + N_OUT * TG_BARS * 8 + 16 + 1024;           // + alignment slack

struct TgBars {
    unsigned long long *a_full, *a_empty, *b_full, *b_empty, *in_full, *in_empty, *acc_full, *acc_empty;
    __device__ TgBars(unsigned char* smem, int o) {
        a_full = reinterpret_cast<unsigned long long*>(smem + TG_OFF_BAR) + o * TG_BARS;
        a_empty = a_full + TG_SETS; b_full = a_empty + TG_SETS; b_empty = b_full + TG_B;
        in_full = b_empty + TG_B; in_empty = in_full + TG_IN_MAX; acc_full = in_empty + TG_IN_MAX; acc_empty = acc_full + TG_BUFS;
    }
};

// Time of a tile.  Measured, 64x(0e+1o+2e) with 0e+1o+2e: 2 150, 2 930 and 3 370 cycles for 6, 8 and 8 slices of 1, 3 and 5 components; with 0e,
// one output, 1 / 2 / 4 slices: 1 100-1 400 / 1 300 / 1 400-1 550 of one component, 1 300-1 600 / 1 600 / 2 050 of three, 1 500 / 1 800 / 2 250 of five (up to a third
// less than the estimate, but alike for the outputs of a problem: none of 18 with several outputs is slower than in the wider kernel for it).
constexpr int tg_cost(int o) { return ts_slices(o) ? 22 * OUT_D[o] + 15 * ts_slices(o) + 103 : 0; }

// matrix descriptor: MN-major, 128-byte rows with 32-byte atoms; blocks of 32 channels `block` bytes apart, four rows 512 bytes
__device__ __forceinline__ unsigned long long tg_desc(unsigned smem_addr, int block) {
    return (unsigned long long)((smem_addr >> 4) & 0x3fff) | (unsigned long long)(block >> 4) << 16 | (unsigned long long)(512 >> 4) << 32 |
           1ull << 46 | 1ull << 61;
}
constexpr unsigned TG_MN_MAJOR = 1u << 15 | 1u << 16;           // instruction descriptor: both operands

// Zeros in the rows of a tile past the batch: they take part in the sums.
template <int O>
__device__ __forceinline__ void tg_zero_rows(unsigned char* in, int rows, int tid, int threads) {
    float *x = reinterpret_cast<float*>(in), *z = reinterpret_cast<float*>(in + TG_X_BYTES), *y = reinterpret_cast<float*>(in + tg_y_at(O));
    for (int i = rows * X_DIM + tid; i < TG_ROWS * X_DIM; i += threads) x[i] = 0.f;
    for (int i = rows * tg_z_len(O) + tid; i < TG_ROWS * tg_z_len(O); i += threads) z[i] = 0.f;
    for (int i = rows * Y_DIM + tid; i < TG_ROWS * Y_DIM; i += threads) y[i] = 0.f;
}
// Inputs of a tile by every thread (arrays that do not start on a 16-byte boundary).
template <int O>
__device__ __forceinline__ void tg_copy_plain(const UvwTsDwParams& p, unsigned char* in, int tile, int tid) {
    constexpr int LEN = tg_z_len(O), THREADS = (TG_PW + TG_BW) * 32;
    const long long row0 = (long long)tile * TG_ROWS;
    const int rows = (int)(p.batch - row0 < TG_ROWS ? p.batch - row0 : TG_ROWS);
    for (int i = tid; i < rows * X_DIM; i += THREADS) reinterpret_cast<float*>(in)[i] = __ldg(p.X + row0 * X_DIM + i);
    for (int i = tid; i < rows * LEN; i += THREADS)
        reinterpret_cast<float*>(in + TG_X_BYTES)[i] = __ldg(p.dZ + (row0 + i / LEN) * Z_DIM + OUT_OFF[O] + i % LEN);
    for (int i = tid; i < rows * Y_DIM; i += THREADS) reinterpret_cast<float*>(in + tg_y_at(O))[i] = __ldg(p.Y + row0 * Y_DIM + i);
    if (rows < TG_ROWS) tg_zero_rows<O>(in, rows, tid, THREADS);
}
// The same as bulk copies, by two warps.
template <int O>
__device__ __forceinline__ void tg_copy_bulk(const UvwTsDwParams& p, unsigned char* in, unsigned long long* full, int tile, unsigned leader, int warp, int lane) {
    constexpr int LEN = tg_z_len(O), EACH = TG_ROWS / 2;
    const long long row0 = (long long)tile * TG_ROWS;
    const int rows = (int)(p.batch - row0 < TG_ROWS ? p.batch - row0 : TG_ROWS);
    const bool all = rows == TG_ROWS;
    if (!all && warp == 0) {                    // (a part of the rows of Y need not be whole 16-byte pieces)
        tg_zero_rows<O>(in, rows, lane, 32);
        for (int i = lane; i < rows * Y_DIM; i += 32) reinterpret_cast<float*>(in + tg_y_at(O))[i] = __ldg(p.Y + row0 * Y_DIM + i);
        __syncwarp();
    }
    const int r0 = warp * EACH, mine = rows - r0 < 0 ? 0 : (rows - r0 < EACH ? rows - r0 : EACH);
    expect_tx_if(leader, full, (unsigned)(mine * (X_DIM + LEN) * 4 + (all && warp == 0 ? TG_Y_BYTES : 0)));
    if (mine > 0) bulk_g2s_if(leader, in + r0 * X_DIM * 4, p.X + (row0 + r0) * X_DIM, (unsigned)(mine * X_DIM * 4), full);
    for (int r = r0; r < r0 + mine; ++r) bulk_g2s_if(leader, in + TG_X_BYTES + r * LEN * 4, p.dZ + (row0 + r) * Z_DIM + OUT_OFF[O], LEN * 4, full);
    if (all && warp == 0) bulk_g2s_if(leader, in + tg_y_at(O), p.Y + row0 * Y_DIM, TG_Y_BYTES, full);
}

// Inputs of a tile: waits for their copy, or takes part in it.  `it`: number of the tile within the CTA's run.
template <int O>
__device__ __forceinline__ bool tg_inputs(const UvwTsDwParams& p, unsigned char* in, const TgBars& bars, int tile, int it, bool ok, int tid) {
    if (p.in_vec) return warp_wait(ok, bars.in_full + it % tg_ins(O), (unsigned)(it / tg_ins(O)) & 1, p.status, ERR_TG_IN);
    tg_copy_plain<O>(p, in, tile, tid);         // (what was in this buffer has been read: the barrier of the tile between)
    group_sync(1, (TG_PW + TG_BW) * 32);
    return ok;
}

// ---------------------------------------------------------------------------- sums
// Row l of MMA tile m is input channel l mod 32 of slice 4 m + l / 32.  Set m of the warps that form T adds the accumulators of a
// segment, columns [hi.hi + lo.hi | hi.lo], to the sums; a warp has a quarter of the rows and every other 16 columns.
template <int O>
__device__ __forceinline__ bool tg_add(const UvwTsDwParams& p, const TgBars& bars, bool ok, unsigned tmem_base, int set, int w, int lane, int segment) {
    constexpr int MW = OUT_MUL[O], MT = tg_mtiles(O);
    if (set >= MT) return ok;
    const unsigned quarter = tmem_base + ((unsigned)((w & 3) * 32) << 16);
    const int n = segment * MT + set, buf = n % TG_BUFS;
    ok = warp_wait(ok, bars.acc_full + buf, (unsigned)(n / TG_BUFS) & 1, p.status, ERR_TG_ACC_FULL);
    if (ok) {
        tc_fence_after();
#pragma unroll 1
        for (int w0 = 16 * (w >> 2); w0 < MW; w0 += 32) {
            const unsigned sum_at = quarter + (unsigned)(128 * TG_BUFS + 64 * set + w0);
            unsigned a[16], b[16];
            tc_load16(quarter + (unsigned)(128 * buf + w0), a);
            tc_load16(quarter + (unsigned)(128 * buf + MW + w0), b);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
            if (segment > 0) {
                tc_load16(sum_at, b);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 16; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
            }
            tc_store16(sum_at, a);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bars.acc_empty + buf);
    return ok;
}

// The sums of the CTA's run of tiles (those of the calling warp).
template <int O>
__device__ __forceinline__ void tg_store(const UvwTsDwParams& p, unsigned tmem_base, int set, int w, int lane) {
    constexpr int MW = OUT_MUL[O];
    if (set >= tg_mtiles(O)) return;
    int from, to;
    ts_ctas<O, tg_cost>(gridDim.x, p.most, from, to);
    float* out = p.ws + (long long)((int)blockIdx.x - from) * W_NUMEL;
    const int slice = 4 * set + (w & 3);
#pragma unroll 1
    for (int w0 = 16 * (w >> 2); w0 < MW; w0 += 32) {
        unsigned v[16];
        tc_load16(tmem_base + ((unsigned)((w & 3) * 32) << 16) + (unsigned)(128 * TG_BUFS + 64 * set + w0), v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            if constexpr (I_OUT[P] == O) {
                constexpr int MU = IN1_MUL[I_IN1[P]], C0 = ts_column(P) / 32;
                const int u = 32 * (slice - C0) + lane;
                if (slice >= C0 && slice < C0 + ts_halves(P) && u < MU) {
                    float* dst = out + W_OFF[P] + weight_offset_v1(MU, MW, u, w0);         // (16 channels of one chunk)
#pragma unroll
                    for (int c = 0; c < 16; ++c) dst[c] = __uint_as_float(v[c]);
                }
            }
        });
    }
}

// ---------------------------------------------------------------------------- T
template <int O>
__device__ __forceinline__ void tg_produce(const UvwTsDwParams& p, unsigned char* smem, const TgBars& bars, int tile_lo, int tile_hi, bool& ok,
                                           unsigned tmem_base, int warp, int lane) {
    constexpr int MT = tg_mtiles(O), BLOCK = tg_block(O), INS = tg_ins(O);
    const int set = warp / TG_SET, w = warp % TG_SET, r = lane & 7;
    // Eight lanes with eight batch rows take the channels of a slice in the order j ^ r: they read eight places of the rows of X (an odd
    // number of pieces apart) and, with the atoms' swizzle r & 3, write eight pieces.
    const int group = (((w & 1) * 4 + (lane >> 3)) ^ r);
    unsigned char* dst = smem + set * tg_a_slot(O) + (w >> 1) * BLOCK + r * 128 + ((group * 16) ^ ((r & 3) << 5));
    int slot_it = 0;                            // slots of all sets so far
    int segment = 0;
    for (int tile = tile_lo, it = 0; tile < tile_hi; ++tile, ++it) {
        unsigned char* in = smem + tg_off_in(O) + it % INS * tg_in(O);
        ok = tg_inputs<O>(p, in, bars, tile, it, ok, warp * 32 + lane);
        const float* x_row = reinterpret_cast<const float*>(in) + r * X_DIM;
        const float* y_row = reinterpret_cast<const float*>(in + tg_y_at(O)) + r * Y_DIM;
        float y_regs[Y_DIM <= 16 ? Y_DIM : 1] = {};
        if constexpr (Y_DIM <= 16) {
#pragma unroll
            for (int j = 0; j < Y_DIM; ++j) y_regs[j] = y_row[j];
        }
        auto y = [&](int j) { return Y_DIM <= 16 ? y_regs[Y_DIM <= 16 ? j : 0] : y_row[j]; };
        for (int mt = 0; mt < MT; ++mt, ++slot_it) {
            if (slot_it % TG_SETS != set) continue;
            const int use = slot_it / TG_SETS, slice = mt * 4 + (w >> 1);
            if (use > 0) ok = warp_wait(ok, bars.a_empty + set, (unsigned)(use - 1) & 1, p.status, ERR_TG_EMPTY);
            if (ok) {
                sfor<0, N_INSTR>([&](auto p_) {
                    constexpr int P = p_;
                    if constexpr (I_OUT[P] == O) {
                        constexpr int A = I_IN1[P], D1 = IN1_D[A], MU = IN1_MUL[A], C0 = ts_column(P) / 32;
                        if (slice >= C0 && slice < C0 + ts_halves(P)) {
                            const int u0 = 32 * (slice - C0) + 4 * group;
                            float x[4 * D1];
#pragma unroll
                            for (int c = 0; c < D1; ++c) {
                                const float4 q = MU % 32 == 0 || u0 < MU ? *reinterpret_cast<const float4*>(x_row + IN1_OFF[A] + u0 * D1 + 4 * c)
                                                                         : make_float4(0.f, 0.f, 0.f, 0.f);
                                x[4 * c] = q.x; x[4 * c + 1] = q.y; x[4 * c + 2] = q.z; x[4 * c + 3] = q.w;
                            }
                            ts_form<P>(x, y, [&](auto k_, float4 hi, float4 lo) {
                                constexpr int K = k_;
                                *reinterpret_cast<float4*>(dst + K * 1024) = hi;
                                *reinterpret_cast<float4*>(dst + K * 1024 + 4 * BLOCK) = lo;
                            });
                        }
                    }
                });
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bars.a_full + set);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.in_empty + it % INS);
        // (a segment's sums are moved when its MMAs are done: where it ends would take registers to know here, 415 us instead of 372)
        const int n = segment * MT + set;
        if (set < MT && __any_sync(0xffffffffu, mbar_test(bars.acc_full + n % TG_BUFS, (unsigned)(n / TG_BUFS) & 1)))
            ok = tg_add<O>(p, bars, ok, tmem_base, set, w, lane, segment++);
    }
    for (const int segments = TgSegments(p.batch, tile_lo).count(p.batch, tile_hi); segment < segments; ++segment)
        ok = tg_add<O>(p, bars, ok, tmem_base, set, w, lane, segment);
    if (ok) tg_store<O>(p, tmem_base, set, w, lane);
}

// ---------------------------------------------------------------------------- dZ, input copies, results
// Two warps split dZ, two copy the inputs as soon as a buffer has been read.
template <int O>
__device__ __forceinline__ void tg_split(const UvwTsDwParams& p, unsigned char* smem, const TgBars& bars, int tile_lo, int tile_hi, bool& ok,
                                         unsigned leader, int warp, int lane) {
    constexpr int D3 = OUT_D[O], MW = OUT_MUL[O], BLOCK = tg_block(O), INS = tg_ins(O);
    const int member = warp & 1, r = lane & 7, group = (member * 4 + (lane >> 3)) ^ r;
    if (warp >= 2 && p.in_vec) {
        for (int tile = tile_lo, it = 0; tile < tile_hi && ok; ++tile, ++it) {
            const int b = it % INS, use = it / INS;
            if (use > 0) ok = warp_wait(ok, bars.in_empty + b, (unsigned)(use - 1) & 1, p.status, ERR_TG_IN_EMPTY);
            if (ok) tg_copy_bulk<O>(p, smem + tg_off_in(O) + b * tg_in(O), bars.in_full + b, tile, leader, member, lane);
        }
        return;
    }
    auto place = [&](int n) { return (n >> 5) * BLOCK + r * 128 + (((n & 31) * 4) ^ ((r & 3) << 5)); };
    for (int tile = tile_lo, it = 0; tile < tile_hi; ++tile, ++it) {
        unsigned char* in = smem + tg_off_in(O) + it % INS * tg_in(O);
        ok = tg_inputs<O>(p, in, bars, tile, it, ok, (TG_PW + warp) * 32 + lane);
        if (warp >= 2) continue;
        const int s = it % TG_B, use = it / TG_B;
        if (use > 0) ok = warp_wait(ok, bars.b_empty + s, (unsigned)(use - 1) & 1, p.status, ERR_TG_B_EMPTY);
        if (ok) {
            unsigned char* slot = smem + tg_off_b(O) + s * tg_b_slot(O);
            sfor<0, (MW + 31) / 32>([&](auto b_) {
                const int w0 = 32 * b_ + 4 * group;         // four output channels
                if (MW % 32 == 0 || w0 < MW) {
                    const float* z = reinterpret_cast<const float*>(in + TG_X_BYTES) + r * tg_z_len(O) + w0 * D3;
                    float v[4 * D3];
#pragma unroll
                    for (int c = 0; c < D3; ++c) {
                        const float4 q = *reinterpret_cast<const float4*>(z + 4 * c);
                        v[4 * c] = q.x; v[4 * c + 1] = q.y; v[4 * c + 2] = q.z; v[4 * c + 3] = q.w;
                    }
                    unsigned char *hi_at = slot + place(w0), *lo_at = slot + place(MW + w0);
#pragma unroll
                    for (int k = 0; k < D3; ++k) {
                        float hi[4], lo[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            hi[u] = tf32_hi(v[u * D3 + k]);
                            lo[u] = v[u * D3 + k] - hi[u];
                        }
                        *reinterpret_cast<float4*>(hi_at + k * 1024) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                        *reinterpret_cast<float4*>(lo_at + k * 1024) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                    }
                }
            });
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bars.b_full + s);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.in_empty + it % INS);
    }
}

// ---------------------------------------------------------------------------- MMA issuer (one warp)
template <int O>
__device__ __forceinline__ void tg_mma(const UvwTsDwParams& p, unsigned char* smem, const TgBars& bars, int tile_lo, int tile_hi, bool& ok,
                                       unsigned tmem_base, unsigned leader) {
    constexpr int D3 = OUT_D[O], MW = OUT_MUL[O], MT = tg_mtiles(O), BLOCK = tg_block(O);
    constexpr unsigned IDESC = tc_instr_desc(MW) | TG_MN_MAJOR, IDESC_WIDE = tc_instr_desc(2 * MW) | TG_MN_MAJOR;
    const unsigned long long a0 = tg_desc(smem_u32(smem), BLOCK), b0 = tg_desc(smem_u32(smem) + tg_off_b(O), BLOCK);
    int slot_it = 0;
    bool ready = false;                         // slot `slot_it` was seen to be full
    bool first = true;
    int segment = 0;                            // (kept apart, and steps by votes: what the MMAs' operands depend on is uniform)
    TgSegments segments(p.batch, tile_lo);
    for (int tile = tile_lo, it = 0; tile < tile_hi && ok; ++tile, ++it) {
        const int s = it % TG_B;
        const bool last = __any_sync(0xffffffffu, tile + 1 == segments.next || tile + 1 == tile_hi);
        ok = warp_wait(ok, bars.b_full + s, (unsigned)(it / TG_B) & 1, p.status, ERR_TG_B_FULL);
        const unsigned long long b = b0 + (unsigned long long)((s * tg_b_slot(O)) >> 4);
#pragma unroll 1
        for (int mt = 0; mt < MT && ok; ++mt, ++slot_it) {
            const int set = slot_it % TG_SETS, n = segment * MT + mt, buf = n % TG_BUFS;
            if (first && n >= TG_BUFS) ok = warp_wait(ok, bars.acc_empty + buf, (unsigned)(n / TG_BUFS - 1) & 1, p.status, ERR_TG_ACC_EMPTY);
            if (!ready) ok = warp_wait(ok, bars.a_full + set, (unsigned)(slot_it / TG_SETS) & 1, p.status, ERR_TG_FULL);
            if (!ok) break;
            tc_fence_after();
            ready = mbar_test(bars.a_full + (slot_it + 1) % TG_SETS, (unsigned)((slot_it + 1) / TG_SETS) & 1);
            const unsigned long long a = a0 + (unsigned long long)((set * tg_a_slot(O)) >> 4);
            const unsigned tmem_d = tmem_base + (unsigned)(128 * buf);
#pragma unroll
            for (int k = 0; k < D3; ++k) {
                tc_mma_if(leader, tmem_d, a + 64 * k, b + 64 * k, IDESC_WIDE, !first || k > 0);                 // [hi.hi | hi.lo]
                tc_mma_if(leader, tmem_d, a + 64 * k + (4 * BLOCK >> 4), b + 64 * k, IDESC, 1);                 // lo.hi
            }
            tc_commit_if(leader, bars.a_empty + set);
            if (last) tc_commit_if(leader, bars.acc_full + buf);
            ready = __all_sync(0xffffffffu, ready);
        }
        if (ok) tc_commit_if(leader, bars.b_empty + s);
        if (last) {
            ++segment;
            segments.advance(p.batch);
        }
        first = last;
    }
}

__device__ void uvw_ts_dw(const UvwTsDwParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + TG_OFF_BAR + N_OUT * TG_BARS * 8);
    if (tid == 0) {
        for (int o = 0; o < N_OUT; ++o) {
            const TgBars bars(smem, o);
            for (int i = 0; i < TG_SETS; ++i) {
                mbar_init(bars.a_full + i, TG_SET);
                mbar_init(bars.a_empty + i, 1);
            }
            for (int i = 0; i < TG_B; ++i) {
                mbar_init(bars.b_full + i, 2);
                mbar_init(bars.b_empty + i, 1);
            }
            for (int i = 0; i < TG_IN_MAX; ++i) {
                mbar_init(bars.in_full + i, 2);
                mbar_init(bars.in_empty + i, TG_PW + 2);
            }
            for (int i = 0; i < TG_BUFS; ++i) {
                mbar_init(bars.acc_full + i, 1);
                mbar_init(bars.acc_empty + i, TG_SET);
            }
        }
        fence_mbar_init();
    }
    if (warp == TG_PW + TG_BW) {        // the MMA warp owns the tensor memory allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TG_COLS) : "memory");
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
            ts_deal<O, TG_ROWS, tg_cost>(p.batch, blockIdx.x, gridDim.x, p.most, lo, hi);
            if (lo < hi) {
                const TgBars bars(smem, O);
                if (warp < TG_PW) {
                    tg_produce<O>(p, smem, bars, lo, hi, ok, tmem_base, warp, lane);
                } else if (warp < TG_PW + TG_BW) {
                    tg_split<O>(p, smem, bars, lo, hi, ok, leader, warp - TG_PW, lane);
                } else {
                    tg_mma<O>(p, smem, bars, lo, hi, ok, tmem_base, leader);
                }
                fence_async_smem();         // (what was an operand may be the destination of bulk copies next)
                tc_fence_before();
                ok = __syncthreads_and(ok);     // (the output is complete: its shared and tensor memory are free)
                tc_fence_after();
            }
        }
    });
    tc_fence_before();
    __syncthreads();
    if (warp == TG_PW + TG_BW)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TG_COLS) : "memory");
}

}  // namespace oeq

#define OEQ_K_UVW_TS_DW 23

extern "C" __global__ void __launch_bounds__(oeq::TG_THREADS, 1) oeq_uvw_ts_dw_kernel(const oeq::UvwTsDwParams p) { oeq::uvw_ts_dw(p); }

// Fixed-order sum of the partial weight gradients of the CTAs.  A weight's output irrep has n of them; with fewer tiles than those,
// tile j is CTA ceil((j + 1) n / tiles) - 1's.  Bound by the latency of the loads, eight in flight: with every
// CTA's run looked up by a thread of every block it took 8.7 us at 1 000 rows, now 7.1, and 5.4 / 3.5 at 20.
extern "C" __global__ void __launch_bounds__(256) oeq_ts_reduce(const float* __restrict__ ws, float* __restrict__ out, long long batch, int ctas, int most) {
    using namespace oeqd;
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    int o = 0, from = 0, to = 0;
    oeq::sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        if (i >= W_OFF[P]) o = I_OUT[P];        // (paths in the order of their weights)
    });
    oeq::sfor<0, N_OUT>([&](auto o_) {
        constexpr int O = o_;
        if constexpr (oeq::ts_slices(O) > 0)
            if (o == O) oeq::ts_ctas<O, oeq::tg_cost>(ctas, most, from, to);
    });
    const long long all = (batch + oeq::TG_ROWS - 1) / oeq::TG_ROWS;
    const int n = to - from, tiles = all < n ? (int)all : n;
    float s = 0.f;
    if (i < W_NUMEL && tiles == n) {
#pragma unroll 8
        for (int j = row; j < tiles; j += 8) s += ws[(long long)j * W_NUMEL + i];
    } else if (i < W_NUMEL) {
#pragma unroll 8
        for (int j = row; j < tiles; j += 8) s += ws[(long long)(((j + 1) * n + tiles - 1) / tiles - 1) * W_NUMEL + i];
    }
    part[row][lane] = s;
    __syncthreads();
    if (row == 0 && i < W_NUMEL) {
#pragma unroll
        for (int r = 1; r < 8; ++r) s += part[r][lane];
        out[i] = s;
    }
}
