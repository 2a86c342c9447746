// Weight gradient of the "uvw" product on the 5th-generation tensor cores (tcgen05, TMEM accumulators), FP32 in / FP32
// out with 3xTF32 error compensation, for shared weights and second-input multiplicity 1:
//
//   dW_p[u,w] = sum_{b,k} T_p[b,u,k] * dZ[b,o,w,k]          (K = batch x components)
//
// with T_p[b,u,k] = sum_{ij} C_p[i,j,k] x[b,u,i] y[b,j] as in the forward pass.  A GEMM whose operands do not exist
// in memory in the needed layout: producer warps build them as K-major, 128-byte-swizzled [rows x 32] tiles split into
// TF32 hi and lo parts, one warp issues the MMAs, and epilogue warps drain tensor memory.  hi.hi and hi.lo go out as
// one MMA over a B tile of 2 N rows (hi tile followed by lo tile), lo.hi as a second one, because issuing an MMA costs
// more than running it.  (dX and dY: dT = W dZ with the forward kernel on the transposed weights, then the channel-wise
// backward kernel on dT.)
//
// Replaces the uvw branches of the reference's backward kernel and its warp-level matmul
// (openequivariance/templates/loop_unroll_tp.cuh:176-219, openequivariance/templates/wmm.cuh:1-88).
// Every wait is bounded; on expiry the role records a code in *status and stops, and the CTA still frees
// its tensor memory.
#pragma once
#include "oeq_common.cuh"
#include "tc_common.cuh"

namespace oeq {
using namespace oeqd;

struct UvwTcBwdParams {
    const float* X;
    const float* Y;
    const float* dZ;
    float* ws;              // [gridDim.x][W_NUMEL] partial weight gradients (dW kernel)
    long long batch;
    int* status;
};

constexpr int TB_EPILOGUE_WARPS = 4;
constexpr int TB_TILE = 128 * 128;             // one [128 rows x 32 tf32] swizzled tile
constexpr int ERR_TB_EMPTY = 31, ERR_TB_FULL = 32, ERR_TB_ACC_EMPTY = 33, ERR_TB_ACC_FULL = 34;

// rows of the batch owned by this CTA
__device__ __forceinline__ void tb_row_range(long long batch, long long& lo, long long& hi) {
    lo = batch * blockIdx.x / gridDim.x;
    hi = batch * (blockIdx.x + 1) / gridDim.x;
}

// ---- paths into an output irrep, grouped so that a group's first-input channels fill the 128 rows of an MMA
constexpr int tb_paths_into(int o) {
    int n = 0;
    for (int p = 0; p < N_INSTR; ++p) n += I_OUT[p] == o;
    return n;
}
constexpr int tb_nth_path(int o, int n) {      // n-th path into o, or -1
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o) {
            if (n == 0) return p;
            --n;
        }
    return -1;
}
constexpr int tb_slot(int o) {                 // rows per path inside a group: 64 if every path is that narrow
    for (int p = 0; p < N_INSTR; ++p)
        if (I_OUT[p] == o && IN1_MUL[I_IN1[p]] > 64) return 128;
    return 64;
}
constexpr int tb_per_group(int o) { return 128 / tb_slot(o); }
constexpr int tb_groups(int o) { return (tb_paths_into(o) + tb_per_group(o) - 1) / tb_per_group(o); }
constexpr int tb_mw_max() {
    int m = 16;
    for (int o = 0; o < N_OUT; ++o) m = OUT_MUL[o] > m ? OUT_MUL[o] : m;
    return m;
}
constexpr int TB_MW_MAX = tb_mw_max();

// =====================================================================================================
// dW kernel.  Per output irrep o and group of paths: D[(path,u), w] += sum over the CTA's batch rows.
// A stage holds RB = floor(32 / (2l+1)) batch rows: A = T^T as [128 (path,u) x 32 (row,k)], B = dZ^T as
// [MW w x 32 (row,k)], both hi and lo.  Every element of a stage is written (value or zero) each time.
// =====================================================================================================
constexpr int DW_B_HALF = TB_MW_MAX * 128;                       // [MW x 32] tile
constexpr int DW_STAGE_BYTES = 2 * TB_TILE + 2 * DW_B_HALF;      // A hi, A lo, B hi, B lo
constexpr int DW_STAGES = (200 * 1024) / DW_STAGE_BYTES < 4 ? (200 * 1024) / DW_STAGE_BYTES : 4;
// One set of four producer warps per stage of the ring: a set builds the same slot every time, so it meets every phase of
// that slot's `empty` barrier.  (A set that changed slots would wait for the parity of a phase without having seen the one
// before it: the wait can pass one phase early, while the tensor core still reads the slot.)
constexpr int TB_PRODUCER_WARPS = 4 * DW_STAGES;
constexpr int TB_THREADS = (TB_PRODUCER_WARPS + 1 + TB_EPILOGUE_WARPS) * 32;
constexpr int DW_ACC_COLS = 2 * TB_MW_MAX;                       // [hi.hi + lo.hi | hi.lo]
constexpr int DW_TMEM_COLS = 2 * DW_ACC_COLS <= 32 ? 32 : 2 * DW_ACC_COLS <= 64 ? 64 : 2 * DW_ACC_COLS <= 128 ? 128
                             : 2 * DW_ACC_COLS <= 256 ? 256 : 512;
constexpr int DW_OFF_BAR = DW_STAGES * DW_STAGE_BYTES;
constexpr int DW_SMEM_BYTES = DW_OFF_BAR + (2 * DW_STAGES + 4) * 8 + 16 + 1024;   // + alignment slack
static_assert(DW_STAGES >= 2, "two stages of the dW kernel must fit in shared memory");
static_assert(2 * TB_MW_MAX <= 256, "output multiplicity above 128");

struct DwBars {
    unsigned long long *full, *empty, *acc_full, *acc_empty;
    unsigned* tmem_slot;
    __device__ explicit DwBars(unsigned char* smem) {
        unsigned long long* b = reinterpret_cast<unsigned long long*>(smem + DW_OFF_BAR);
        full = b; empty = b + DW_STAGES; acc_full = b + 2 * DW_STAGES; acc_empty = acc_full + 2;
        tmem_slot = reinterpret_cast<unsigned*>(acc_empty + 2);
    }
};

// Four rows of values v[row][k] of a tile row (slot row or output channel): columns (4 g + row) D3 + k, which are whole
// 16-byte pieces, split into hi and lo.  Rows the stage does not have are zeros, so every column of a tile is written.
template <int D3>
__device__ __forceinline__ void dw_store4(unsigned char* hi_row, int lo_off, int row, int g, const float (&v)[4][D3]) {
#pragma unroll
    for (int c = 0; c < D3; ++c) {
        const int piece = g * D3 + c;
        if (piece < 8) {
            float h[4], l[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float t = v[(4 * c + i) / D3][(4 * c + i) % D3];
                h[i] = tf32_hi(t);
                l[i] = t - h[i];
            }
            unsigned char* dst = hi_row + ((piece ^ (row & 7)) << 4);
            *reinterpret_cast<float4*>(dst) = make_float4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<float4*>(dst + lo_off) = make_float4(l[0], l[1], l[2], l[3]);
        }
    }
}

// Bound by issue: with a thread per (slot row, every fourth batch row) each element paid a swizzled address and two
// 4-byte stores.  Four warps now build a whole stage (one set of warps per slot of the ring): a thread keeps one slot
// row and walks the stage's batch rows four at a time, whose values fill whole 16-byte pieces.
template <int O, int GRP>
__device__ __forceinline__ bool dw_produce(const UvwTcBwdParams& p, unsigned char* smem, const DwBars& bars,
                                           long long row_lo, long long row_hi, long long& stage_it, int ptid) {
    constexpr int D3 = OUT_D[O], RB = 32 / D3, MW = OUT_MUL[O];
    constexpr int SLOT = tb_slot(O), PER = tb_per_group(O);
    constexpr int GROUPS = (8 + D3 - 1) / D3;           // groups of four rows that cover the 32 columns
    const int set = ptid >> 7, t = ptid & 127;
    const int which = t / SLOT, u = t % SLOT;
    bool ok = true;
    for (long long b0 = row_lo; b0 < row_hi && ok; b0 += RB, ++stage_it) {
        const int s = (int)(stage_it % DW_STAGES);
        if (s != set) continue;
        const int rows = (int)(row_hi - b0 < RB ? row_hi - b0 : RB);
        const long long use = stage_it / DW_STAGES;
        if (use > 0) ok = mbar_wait(bars.empty + s, (unsigned)((use - 1) & 1), p.status, ERR_TB_EMPTY);
        if (!ok) break;
        unsigned char* a_hi = smem + s * DW_STAGE_BYTES;
        unsigned char* b_hi = a_hi + 2 * TB_TILE;       // the lo tile follows the hi tile: one descriptor spans both
        // ---- A: T^T, slot row t = (path, u)
        unsigned char* a_row = a_hi + (t >> 3) * 1024 + (t & 7) * 128;
        bool done = false;
        sfor<0, PER>([&](auto j_) {
            constexpr int P = tb_nth_path(O, GRP * PER + j_);
            if constexpr (P >= 0) {
                constexpr int a = I_IN1[P], b = I_IN2[P], D1 = IN1_D[a], D2 = IN2_D[b], MU = IN1_MUL[a];
                if (which == j_ && u < MU) {
                    done = true;
                    const float* x0 = p.X + b0 * X_DIM + IN1_OFF[a] + u * D1;
                    const float* y0 = p.Y + b0 * Y_DIM + IN2_OFF[b];
#pragma unroll 1
                    for (int g = 0; g < GROUPS; ++g) {
                        float x[4][D1], y[4][D2], v[4][D3];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const bool live = 4 * g + q < rows;
                            const float* xr = x0 + (4 * g + q) * X_DIM;
                            const float* yr = y0 + (4 * g + q) * Y_DIM;
#pragma unroll
                            for (int i = 0; i < D1; ++i) x[q][i] = live ? __ldg(xr + i) : 0.f;
#pragma unroll
                            for (int j = 0; j < D2; ++j) y[q][j] = live ? __ldg(yr + j) : 0.f;
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
#pragma unroll
                            for (int k = 0; k < D3; ++k) v[q][k] = 0.f;
                            float xy = 0.f;
                            sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                                constexpr int N = n_;
                                if constexpr (N == CG_BEGIN[P] || CG_I[N] != CG_I[N - 1] || CG_J[N] != CG_J[N - 1])
                                    xy = x[q][CG_I[N]] * y[q][CG_J[N]];
                                v[q][CG_K[N]] = fmaf(xy, (float)CG_V[N], v[q][CG_K[N]]);
                            });
                        }
                        dw_store4<D3>(a_row, TB_TILE, t, g, v);
                    }
                }
            }
        });
        if (!done) {      // no path in this slot, or a channel beyond its multiplicity: a row of zeros
#pragma unroll
            for (int piece = 0; piece < 8; ++piece) {
                *reinterpret_cast<float4*>(a_row + piece * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(a_row + piece * 16 + TB_TILE) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        // ---- B: dZ^T, one row per output channel; channels fewer than threads: the groups of rows are shared out
        constexpr int WT = MW <= 32 ? 32 : (MW <= 64 ? 64 : 128), PARTS = 128 / WT;
        static_assert(MW <= 128, "output multiplicity above 128");
        const int w = t % WT;
        if (w < MW) {
            unsigned char* b_row = b_hi + (w >> 3) * 1024 + (w & 7) * 128;
            const float* z0 = p.dZ + b0 * Z_DIM + OUT_OFF[O] + w * D3;
#pragma unroll 1
            for (int g = t / WT; g < GROUPS; g += PARTS) {
                float v[4][D3];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int k = 0; k < D3; ++k) v[q][k] = 4 * g + q < rows ? __ldg(z0 + (long long)(4 * g + q) * Z_DIM + k) : 0.f;
                dw_store4<D3>(b_row, MW * 128, w, g, v);
            }
        }
        fence_async_smem();
        __syncwarp();
        if ((ptid & 31) == 0) mbar_arrive(bars.full + s);
    }
    return ok;
}

template <int O, int GRP>
__device__ __forceinline__ bool dw_mma(const UvwTcBwdParams& p, unsigned char* smem, const DwBars& bars, long long row_lo,
                                       long long row_hi, long long& stage_it, long long& acc_it, unsigned tmem_base, unsigned leader) {
    constexpr int D3 = OUT_D[O], RB = 32 / D3, MW = OUT_MUL[O];
    constexpr unsigned IDESC = tc_instr_desc(MW), IDESC_WIDE = tc_instr_desc(2 * MW);
    if (row_lo >= row_hi) return true;
    const int t = (int)(acc_it & 1);
    const long long acc_use = acc_it >> 1;
    if (acc_use > 0 && !warp_wait(true, bars.acc_empty + t, (unsigned)((acc_use - 1) & 1), p.status, ERR_TB_ACC_EMPTY)) return false;
    tc_fence_after();
    const unsigned tmem_d = tmem_base + (unsigned)(t * DW_ACC_COLS);
    const unsigned long long desc0 = tc_smem_desc(smem_u32(smem));
    unsigned accumulate = 0;
    bool ready = false, ahead = false;      // this stage and the next one were seen to be full, two stages ahead
    for (long long b0 = row_lo; b0 < row_hi; b0 += RB) {
        const int s = (int)(stage_it % DW_STAGES);
        const long long use = stage_it / DW_STAGES;
        if (!ready && !warp_wait(true, bars.full + s, (unsigned)(use & 1), p.status, ERR_TB_FULL)) return false;
        tc_fence_after();
        const unsigned long long da_hi = desc0 + (unsigned long long)((s * DW_STAGE_BYTES) >> 4);
        const unsigned long long da_lo = da_hi + (TB_TILE >> 4);
        const unsigned long long db = da_lo + (TB_TILE >> 4);        // hi tile, then lo tile
        const bool asked = DW_STAGES > 2 && mbar_test(bars.full + (stage_it + 2) % DW_STAGES, (unsigned)((stage_it + 2) / DW_STAGES & 1));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            tc_mma_if(leader, tmem_d, da_hi + 2 * kk, db + 2 * kk, IDESC_WIDE, accumulate);   // [hi.hi | hi.lo]
            accumulate = 1;
            tc_mma_if(leader, tmem_d, da_lo + 2 * kk, db + 2 * kk, IDESC, 1);                 // lo.hi into the first half
        }
        tc_commit_if(leader, bars.empty + s);
        ready = __all_sync(0xffffffffu, ahead);
        ahead = asked;
        ++stage_it;
    }
    tc_commit_if(leader, bars.acc_full + t);
    ++acc_it;
    return true;
}

template <int O, int GRP>
__device__ __forceinline__ bool dw_epilogue(const UvwTcBwdParams& p, const DwBars& bars, long long row_lo, long long row_hi,
                                            long long& acc_it, unsigned tmem_base, int ewarp, int lane) {
    constexpr int MW = OUT_MUL[O];
    constexpr int SLOT = tb_slot(O), PER = tb_per_group(O);
    float* out = p.ws + (long long)blockIdx.x * W_NUMEL;
    const int srow = ewarp * 32 + lane, which = srow / SLOT, u = srow % SLOT;
    if (row_lo >= row_hi) {   // no rows: this CTA's slice of the partial gradients is zero
        sfor<0, PER>([&](auto j_) {
            constexpr int P = tb_nth_path(O, GRP * PER + j_);
            if constexpr (P >= 0) {
                if (which == j_ && u < IN1_MUL[I_IN1[P]])
                    for (int w = 0; w < MW; ++w) out[W_OFF[P] + weight_offset_v1(IN1_MUL[I_IN1[P]], MW, u, w)] = 0.f;
            }
        });
        return true;
    }
    const int t = (int)(acc_it & 1);
    const long long use = acc_it >> 1;
    if (!mbar_wait(bars.acc_full + t, (unsigned)(use & 1), p.status, ERR_TB_ACC_FULL)) return false;
    tc_fence_after();
    // accumulator row = (path, u); a warp may only read the TMEM lanes of its own quarter
    const unsigned taddr = tmem_base + ((unsigned)(ewarp * 32) << 16) + (unsigned)(t * DW_ACC_COLS);
#pragma unroll
    for (int c0 = 0; c0 < MW; c0 += 16) {
        unsigned v[16], v2[16];
        tc_load16(taddr + (unsigned)c0, v);
        tc_load16(taddr + (unsigned)(MW + c0), v2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        sfor<0, PER>([&](auto j_) {
            constexpr int P = tb_nth_path(O, GRP * PER + j_);
            if constexpr (P >= 0) {
                if (which == j_ && u < IN1_MUL[I_IN1[P]]) {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        out[W_OFF[P] + weight_offset_v1(IN1_MUL[I_IN1[P]], MW, u, c0 + c)] = __uint_as_float(v[c]) + __uint_as_float(v2[c]);
                }
            }
        });
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bars.acc_empty + t);
    ++acc_it;
    return true;
}

// Small batches: the groups of paths are dealt over the grid's y dimension.
constexpr int dw_groups_before(int o) {
    int n = 0;
    for (int q = 0; q < o; ++q) n += tb_groups(q);
    return n;
}

__device__ void uvw_tc_dw(const UvwTcBwdParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const DwBars bars(smem);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    long long row_lo, row_hi;
    tb_row_range(p.batch, row_lo, row_hi);
    if (tid == 0) {
        for (int i = 0; i < DW_STAGES; ++i) {
            mbar_init(bars.full + i, 4);
            mbar_init(bars.empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bars.acc_full + i, 1);
            mbar_init(bars.acc_empty + i, TB_EPILOGUE_WARPS);
        }
        fence_mbar_init();
    }
    if (warp == TB_PRODUCER_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(bars.tmem_slot)),
                     "n"(DW_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile unsigned*>(bars.tmem_slot), 0);

    if (warp < TB_PRODUCER_WARPS) {
        long long stage_it = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            sfor<0, tb_groups(O)>([&](auto g_) {
                constexpr int GRP = g_;
                if (gridDim.y > 1 && (int)blockIdx.y != dw_groups_before(O) + GRP) return;
                if (ok) ok = dw_produce<O, GRP>(p, smem, bars, row_lo, row_hi, stage_it, tid);
            });
        });
    } else if (warp == TB_PRODUCER_WARPS) {
        const unsigned leader = elect_lane();
        long long stage_it = 0, acc_it = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            sfor<0, tb_groups(O)>([&](auto g_) {
                constexpr int GRP = g_;
                if (gridDim.y > 1 && (int)blockIdx.y != dw_groups_before(O) + GRP) return;
                if (ok) ok = dw_mma<O, GRP>(p, smem, bars, row_lo, row_hi, stage_it, acc_it, tmem_base, leader);
            });
        });
        __syncwarp();
    } else {
        long long acc_it = 0;
        bool ok = true;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int O = o_;
            sfor<0, tb_groups(O)>([&](auto g_) {
                constexpr int GRP = g_;
                if (gridDim.y > 1 && (int)blockIdx.y != dw_groups_before(O) + GRP) return;
                if (ok) ok = dw_epilogue<O, GRP>(p, bars, row_lo, row_hi, acc_it, tmem_base, warp & 3, lane);
            });
        });
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TB_PRODUCER_WARPS) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(DW_TMEM_COLS) : "memory");
    }
}

}  // namespace oeq

#define OEQ_K_UVW_TC_DW 21

extern "C" __global__ void __launch_bounds__(oeq::TB_THREADS, 1) oeq_uvw_tc_dw_kernel(const oeq::UvwTcBwdParams p) {
    oeq::uvw_tc_dw(p);
}

// Fixed-order sum of the partial weight gradients.
extern "C" __global__ void __launch_bounds__(256) oeq_reduce_partials(const float* ws, float* out, int n, long long groups) {
    oeq::reduce_partials(ws, out, n, groups);
}
