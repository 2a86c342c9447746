// Parts that the tensor-core 'uvw' kernels with a batch row per lane share (uvw_ts_kernels.cuh, uvw_ts_dw_kernels.cuh): how
// the work is dealt, copies issued from a warp in step, and T of a row.
#pragma once
#include "tc_common.cuh"

namespace oeq {
using namespace oeqd;

// ---- slices of 32 input channels of the paths into an output irrep, in the order of the paths
constexpr int ts_halves(int p) { return (IN1_MUL[I_IN1[p]] + 31) / 32; }
constexpr int ts_column(int p) {                // input channels, in whole slices, before those of path p
    int n = 0;
    for (int q = 0; q < p; ++q) n += I_OUT[q] == I_OUT[p] ? 32 * ts_halves(q) : 0;
    return n;
}
constexpr int ts_slices(int o) {
    int n = 0;
    for (int p = 0; p < N_INSTR; ++p) n += I_OUT[p] == o ? ts_halves(p) : 0;
    return n;
}

// Tiles of ROWS batch rows: the CTAs are dealt to the output irreps by the time that an output's tiles take, a tile's time being
// COST, and an output's tiles in equal runs to its CTAs (fewer CTAs than outputs take a run of every output).  Code for two outputs
// does not fit the instruction caches: a CTA that goes from one output to the next is 1.4 times slower than the others, and so
// are two CTAs on neighbouring SMs, which are two of consecutive numbers, that work on different ones; hence even bounds.
// No output has more than `most` of them.
template <int O, int (*COST)(int)>
__device__ __forceinline__ void ts_ctas(int ctas, int most, int& from, int& to) {
    int total = 0, outputs = 0;
    sfor<0, N_OUT>([&](auto o_) {
        constexpr int cost = COST(o_);
        total += cost;
        outputs += cost > 0;
    });
    from = 0;
    to = ctas;
    if (ctas >= outputs) {                                  // one CTA or more for every output
        int cost = 0, left = outputs;
        to = 0;
        sfor<0, O + 1>([&](auto o_) {
            constexpr int c = COST(o_);
            if constexpr (c > 0) {
                cost += c;
                --left;
                from = to;
                int at = (int)(((long long)ctas * cost + total / 2) / total);
                if (ctas >= 16 * outputs && left > 0) at = (at + 1) / 2 * 2;
                to = at > from ? at : from + 1;
                to = to < ctas - left ? to : ctas - left;
            }
        });
    }
    to = to - from < most ? to : from + most;
}
template <int O, int ROWS, int (*COST)(int)>
__device__ __forceinline__ void ts_deal(long long batch, int cta, int ctas, int most, int& lo, int& hi) {
    const long long tiles = (batch + ROWS - 1) / ROWS;
    int from, to;
    ts_ctas<O, COST>(ctas, most, from, to);
    const bool mine = cta >= from && cta < to;
    lo = mine ? (int)(tiles * (cta - from) / (to - from)) : 0;
    hi = mine ? (int)(tiles * (cta - from + 1) / (to - from)) : 0;
}

// ---- issued by the lane whose `leader` is set; every lane of the warp comes here
__device__ __forceinline__ void expect_tx_if(unsigned leader, unsigned long long* bar, unsigned bytes) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b64 st;\n\tsetp.ne.b32 q, %2, 0;\n\t"
        "@q mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "r"(bytes), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void bulk_g2s_if(unsigned leader, void* dst_smem, const void* src_gmem, unsigned bytes, unsigned long long* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
        "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(smem_u32(dst_smem)),
        "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar)), "r"(leader)
        : "memory");
}
// 16 columns of the calling warp's 32 TMEM lanes
__device__ __forceinline__ void tc_store16(unsigned taddr, const unsigned* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr)
        : "memory");
}

// ---- T of a batch row: T[u,k] = sum_i M[i,k] x[u,i], M[i,k] = sum_j C_ijk y_j
template <int P, int N> constexpr bool ts_first_entry() {
    for (int m = CG_BEGIN[P]; m < N; ++m)
        if (CG_I[m] == CG_I[N] && CG_K[m] == CG_K[N]) return false;
    return true;
}
template <int P, int N> constexpr bool ts_first_of_k() {
    for (int m = CG_BEGIN[P]; m < N; ++m)
        if (CG_K[m] == CG_K[N]) return false;
    return true;
}

// T of path P for four input channels x[4][2l+1], split into TF32 hi and lo parts: store(k, hi, lo) for every component.  M is
// formed for these four channels alone; y(j) is the row's second input.
template <int P, class YF, class SF>
__device__ __forceinline__ void ts_form(const float (&x)[4 * IN1_D[I_IN1[P]]], YF&& y, SF&& store) {
    constexpr int D1 = IN1_D[I_IN1[P]], D3 = OUT_D[I_OUT[P]], Y0 = IN2_OFF[I_IN2[P]];
    float m[D1][D3];
    sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
        constexpr int N = n_;
        float& e = m[CG_I[N]][CG_K[N]];
        if constexpr (ts_first_entry<P, N>()) e = (float)CG_V[N] * y(Y0 + CG_J[N]);
        else e = fmaf((float)CG_V[N], y(Y0 + CG_J[N]), e);
    });
    sfor<0, D3>([&](auto k_) {
        constexpr int K = k_;
        float t[4] = {0.f, 0.f, 0.f, 0.f}, hi[4], lo[4];
        sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
            constexpr int N = n_, I = CG_I[N];
            if constexpr (CG_K[N] == K && ts_first_entry<P, N>()) {
#pragma unroll
                for (int u = 0; u < 4; ++u) t[u] = ts_first_of_k<P, N>() ? m[I][K] * x[u * D1 + I] : fmaf(m[I][K], x[u * D1 + I], t[u]);
            }
        });
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            hi[u] = tf32_hi(t[u]);
            lo[u] = t[u] - hi[u];               // exact; read as TF32 by the MMA
        }
        store(k_, make_float4(hi[0], hi[1], hi[2], hi[3]), make_float4(lo[0], lo[1], lo[2], lo[3]));
    });
}

}  // namespace oeq
