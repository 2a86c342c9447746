// "uvu" graph convolution for sm_100a, one warp per (run of edges, slice of 32 channels).
//
// The kernels of uvu_kernels.cuh give an edge to a group of warps with a staging warp of its own; per edge the
// group hands a stage over, and one thread issues the bulk copies of X, Y and W one after the other.  Here every
// warp is on its own: it walks edges in receiver order, copies *its* 32 channels of the rows ahead with 16-byte
// cp.async (no staging warp, no barrier wider than a warp, so no third warp on a scheduler caps the registers) and
// takes two edges of one receiver at a time.
//   * FP32: the two edges are the two halves of packed registers.  Products, and the coefficient FMAs of paths that take their
//     weight on the result, are one packed instruction for both edges (fma.rn.f32x2, two cycles of a scheduler's dispatch);
//     where the weight is on an input the coefficient FMAs go straight to the receiver's row, one scalar FMA with an immediate
//     for each edge.
//   * Products x_i y_j are formed once for all paths that share the two input irreps (E_* tables).
//   * FP64: the same code with one edge at a time.
// The walk deals chunks of consecutive edges round robin, so that gathered rows are shared in L2.
// Measured against the group kernels: 32x(0e+1o+2e) on 20 000 nodes / 800 k edges, atomic, forward 463 -> 262 us and
// backward 796 -> 585 us; 128x(0e+1o+2e) x (0e..3o) on 5 000 nodes / 150 k edges, deterministic, 446 -> 297 and 854 -> 585.
#pragma once
#define OEQ_UVU_NO_ENTRY
#include "uvu_kernels.cuh"

#define OEQ_K_SLICE_FWD_DET 50
#define OEQ_K_SLICE_FWD_ATOMIC 51
#define OEQ_K_SLICE_BWD_ATOMIC 53
#define OEQ_K_SLICE_DBL_Z_DET 54
#define OEQ_K_SLICE_DBL_Z_ATOMIC 55

namespace oeq {

constexpr int SL_S = SLICE_STAGES;              // stages per warp
constexpr int SL_WARPS = SLICE_WARPS;           // warps per CTA, a multiple of N_SLICE
constexpr int CPL = SLICE_CPL, CH = 32 * CPL;   // channels per lane and of a slice
constexpr int N_SLICE = NSLICE;                 // slices of a row (1: the whole row)
constexpr bool FULL = SLICE_FULL;               // every multiplicity is CH * NSLICE

// Without weights (UNIT_W) the coefficients are the same for all edges of a receiver, so a run of edges needs only the
// products of the two inputs per edge: forward, the sums B_ij = sum_e x_i y_j are kept and contracted once per receiver;
// backward, G_ij = sum_k C_ijk dZ_k is formed once per receiver.  B and G hold the pairs (i, j) that have a coefficient (PR_I,
// PR_J; GRP_PR: where a pair of irreps starts, CG_PR: the place of a coefficient's pair): a component times the zeros of
// other pairs would be work for nothing, and NaN where it is infinite.
// Edge sums of 64x(0e+1o+2e) x (0e+1o+2e), 10 007 nodes / 400 k edges: forward 265 -> 211 us, backward 433 -> 393 us.  Per
// channel and edge 71 and 142 FMAs instead of 71 products, 83 coefficient FMAs and 35 additions forward, 83 coefficient FMAs for
// two edges and 158 for each backward; the walk, the copies and the sum of dY take 110 and 200 instructions beside them.
constexpr bool OUTER = SLICE_OUTER;
static_assert(CPL == 1 || (OUTER && FULL), "several channels per lane: backward edge sums of full slices");

// ---- two edges in one register pair (FP32), or one edge (FP64, and the forward sums of products)
#if OEQ_KERNEL == OEQ_K_SLICE_FWD_DET || OEQ_KERNEL == OEQ_K_SLICE_FWD_ATOMIC || OEQ_KERNEL == OEQ_K_SLICE_DBL_Z_DET || OEQ_KERNEL == OEQ_K_SLICE_DBL_Z_ATOMIC
constexpr bool FORWARD = true;                  // the walk that sums rows of Z
constexpr bool ONE_EDGE = OUTER || SLICE_ONE || ELEM == 8;   // (packing saves nothing where every product goes into a sum of its own)
#else
constexpr bool FORWARD = false;
constexpr bool ONE_EDGE = CPL > 1 || SLICE_ONE || ELEM == 8;
#endif
template <class U, bool ONE> struct Pack;
template <> struct Pack<float, false> {
    typedef unsigned long long V;
    static constexpr int N = 2;
    static __device__ __forceinline__ V make(float a, float b) { V r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
    static __device__ __forceinline__ float get(V v, int h) {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return h ? b : a;
    }
    static __device__ __forceinline__ V mul(V a, V b) { V r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { V r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
    static __device__ __forceinline__ V add(V a, V b) { V r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
    static __device__ __forceinline__ V all(float c) { return make(c, c); }
};
template <class U> struct Pack<U, true> {
    typedef U V;
    static constexpr int N = 1;
    static __device__ __forceinline__ V make(U a, U) { return a; }
    static __device__ __forceinline__ U get(V v, int) { return v; }
    static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
    static __device__ __forceinline__ V add(V a, V b) { return a + b; }
    static __device__ __forceinline__ V all(U c) { return c; }
};
typedef Pack<T, ONE_EDGE> PK;
typedef PK::V V2;

// ---- slice layout of a stage: X and W of its two edges, or one, and Y (packed pairs: interleaved, element j of edge h at 2j + h)
__host__ __device__ constexpr int sum_in1_d(int n) { int s = 0; for (int a = 0; a < n; ++a) s += IN1_D[a]; return s; }
constexpr int EP = SLICE_ONE ? 1 : 2;                               // edges of a stage
constexpr int X_CH = sum_in1_d(N_IN1);                              // X values per channel
constexpr int XS_ELEMS = FULL ? CH * X_CH : X_DIM;                  // X values of a slice
constexpr int WS_ELEMS = UNIT_W ? 0 : (FULL ? 32 * N_INSTR : W_NUMEL);
constexpr int XSB = pad16(XS_ELEMS * ELEM), WSB = pad16(WS_ELEMS * ELEM), YSB = pad16(EP * Y_DIM * ELEM);
// where irrep a of X, weight p of a slice start
template <int A> __host__ __device__ constexpr int xs_off() { return FULL ? CH * sum_in1_d(A) : IN1_OFF[A]; }
template <int P> __host__ __device__ constexpr int ws_off() { return FULL ? 32 * P : W_OFF[P]; }

struct SliceStage {
    static constexpr int OFF_HDR = 0;           // first edge, receiver, sender of edge 0, sender of edge 1 (-1: one edge)
    static constexpr int OFF_Y = 16;
    static constexpr int OFF_EY = OFF_Y + YSB;  // (second derivatives: the cotangent rows beside the rows)
    static constexpr int OFF_X = OFF_EY + (DBLC ? YSB : 0);     // a row of each edge
    static constexpr int OFF_EX = OFF_X + EP * XSB;
    static constexpr int OFF_W = OFF_EX + (DBLC ? EP * XSB : 0);
    static constexpr int OFF_EW = OFF_W + EP * WSB;
    static constexpr int BYTES = OFF_EW + (DBLC ? EP * WSB : 0);
};
constexpr int MAX_OUT_D = []() { int m = 1; for (int o = 0; o < N_OUT; ++o) m = OUT_D[o] > m ? OUT_D[o] : m; return m; }();
constexpr int SL_FLUSH = pad16(32 * MAX_OUT_D * ELEM);              // transposition buffer of one output irrep

// (`size` of the 16, or ELEM, bytes come from memory, the others are zeros)
__device__ __forceinline__ void cp_async_16_hint(void* dst_smem, const void* src_gmem, int size, unsigned long long policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "r"(size), "l"(policy) : "memory");
}
__device__ __forceinline__ void cp_async_elem_fill(void* dst_smem, const void* src_gmem, int size) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "n"(ELEM), "r"(size) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }


// ---------------------------------------------------------------- walk and staging

// The pairs of edges of one warp, all lanes in step: chunks walker, walker + walkers, ... of consecutive edges in
// receiver order; ALIGN moves chunk ends forward to the next receiver so that a receiver has one writer.
template <bool ALIGN>
struct PairWalker {
    const UvuParams& p;
    int lane, walkers, chunk, n_chunks;
    int pos, end;               // next edge of the chunk, its end
    int wbase;                  // window: lane l holds receiver and sender of edge wbase + l ...
    int wr, wc, nr, nc;         // ... and of edge wbase + 31 + l, fetched ahead
    int node_hi, expect;        // ALIGN: end of the chunk's node range, first node not yet met

    __device__ PairWalker(const UvuParams& p_, int walkers_, int walker, int lane_)
        : p(p_), lane(lane_), walkers(walkers_), chunk(walker - walkers_) {
        n_chunks = (int)((p.n_items + p.chunk - 1) / p.chunk);
        pos = end = 0;
        wbase = wr = wc = nr = nc = node_hi = expect = 0;
    }
    __device__ __forceinline__ void load(int base, int& r, int& c) const {
        const int k = base + lane;
        r = c = -1;
        if (k < end) {
            r = (int)p.rows[k];
            c = (int)p.cols[k];
        }
    }
    // First edge >= t that starts a receiver, given the receivers r of edges t - 1 + lane (-1 past the list).
    __device__ __forceinline__ int align(int t, int r) const {
        const int n = (int)p.n_items;
        if (t <= 0) return 0;
        if (t >= n) return n;
        for (;;) {
            const int before = __shfl_up_sync(0xffffffffu, r, 1);
            const unsigned b = __ballot_sync(0xffffffffu, lane > 0 && r != before);
            if (b) return min(n, t + __ffs(b) - 2);
            t += 31;
            r = receiver(t - 1 + lane);
        }
    }
    __device__ __forceinline__ int receiver(int k) const { return k >= 0 && k < (int)p.n_items ? (int)p.rows[k] : -1; }
    __device__ bool next_chunk() {
        for (;;) {
            chunk += walkers;
            if (chunk >= n_chunks) return false;
            const int n = (int)p.n_items;
            const long long t = (long long)chunk * p.chunk;
            if constexpr (ALIGN) {
                const int t1 = (int)min((long long)n, t + p.chunk);
                const int ra = receiver((int)t - 1 + lane), rb = receiver(t1 - 1 + lane);    // one latency for both ends
                pos = align((int)t, ra);
                end = align(t1, rb);
                if (pos >= end) continue;   // no receiver starts in this chunk
                node_hi = end >= n ? (int)p.n_nodes : receiver(end);
                expect = chunk == 0 ? 0 : -1;
            } else {
                pos = (int)t;
                end = (int)min((long long)n, t + p.chunk);
            }
            wbase = pos;
            load(wbase, wr, wc);
            load(wbase + 31, nr, nc);
            return true;
        }
    }
    // Next pair: first edge, receiver, senders (s1 < 0: the pair has one edge).  ALIGN: the nodes [g0, row) and
    // [row + 1, g1) receive nothing.
    __device__ __forceinline__ bool next(int& e0, int& row, int& s0, int& s1, int& g0, int& g1) {
        if (pos >= end) {
            if (!next_chunk()) return false;
        }
        int src = pos - wbase;
        if (src >= 31) {
            wr = nr;
            wc = nc;
            wbase += 31;
            src -= 31;
            load(wbase + 31, nr, nc);
        }
        row = __shfl_sync(0xffffffffu, wr, src);
        s0 = __shfl_sync(0xffffffffu, wc, src);
        const int r1 = __shfl_sync(0xffffffffu, wr, src + 1), c1 = __shfl_sync(0xffffffffu, wc, src + 1);
        const bool two = EP == 2 && r1 == row;      // (a lane past the chunk holds -1)
        s1 = two ? c1 : -1;
        e0 = pos;
        pos += two ? 2 : 1;
        if constexpr (ALIGN) {
            g0 = expect < 0 ? row : expect;     // (a chunk's first receiver: the nodes before it are the chunk before's)
            expect = row + 1;
            g1 = pos >= end ? node_hi : 0;
        }
        return true;
    }
};

// ---- 16-byte pieces and elements from shared to global memory: stored, or added
__device__ __forceinline__ void red_add_v4(float* dst, float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
template <bool ADD> __device__ __forceinline__ void elem_out(T* dst, T v) {
    if constexpr (ADD) red_add(dst, v);
    else *dst = v;
}
template <bool ADD> __device__ __forceinline__ void piece_out(T* dst, const T* src) {
    if constexpr (!ADD) {
        *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(src);
    } else if constexpr (ELEM == 4) {
        red_add_v4(reinterpret_cast<float*>(dst), *reinterpret_cast<const float4*>(src));
    } else {
        red_add(dst, src[0]);
        red_add(dst + 1, src[1]);
    }
}
template <bool ADD>
__device__ __forceinline__ void row_out(T* dst, const T* src, int n, bool vec, int lane) {
    constexpr int EPV = 16 / ELEM;
    if (vec) {
        for (int q = lane; q < n / EPV; q += 32) piece_out<ADD>(dst + q * EPV, src + q * EPV);
    } else {
        for (int q = lane; q < n; q += 32) elem_out<ADD>(dst + q, src[q]);
    }
}

// Copies of one warp: 16-byte pieces when the arrays allow it, elements otherwise.
struct SliceCopies {
    static constexpr int EPV = 16 / ELEM;
    static constexpr int XQ = XSB / 16, WQ = WSB / 16, XI = (XQ + 31) / 32, WI = (WQ + 31) / 32;
    int xo[FULL && N_SLICE > 1 ? XI : 1];       // element offset in the row of this lane's i-th piece of X
    int slice, lane;
    bool xv, wv;
    unsigned long long keep, stream;
    __device__ SliceCopies(const UvuParams& p, int slice_, int lane_) : slice(slice_), lane(lane_) {
        xv = p.flags & 1;
        wv = p.flags & 4;
        keep = l2_policy_evict_last();
        stream = l2_policy_evict_first();
        if constexpr (FULL && N_SLICE > 1) {
#pragma unroll
            for (int i = 0; i < XI; ++i) {
                const int el = (lane + 32 * i) * EPV;
                int o = 0;
                sfor<0, N_IN1>([&](auto a_) {
                    constexpr int a = a_;
                    constexpr int lo = xs_off<a>(), n = CH * IN1_D[a];
                    if (el >= lo && el < lo + n) o = IN1_OFF[a] + slice * n + (el - lo);
                });
                xo[i] = o;
            }
        }
    }
    __device__ __forceinline__ void x_row(unsigned char* dst, const T* row, bool fill) const {
        const int b16 = fill ? 0 : 16, be = fill ? 0 : ELEM;
        if (xv) {
#pragma unroll
            for (int i = 0; i < XI; ++i) {
                const int q = lane + 32 * i;
                if (32 * i + 32 <= XQ || q < XQ) {
                    if constexpr (FULL && N_SLICE > 1) cp_async_16_hint(dst + 16 * q, row + xo[i], b16, keep);
                    else cp_async_16_hint(dst + 16 * q, row + q * EPV, b16, keep);
                }
            }
        } else if constexpr (FULL && N_SLICE > 1) {
            sfor<0, N_IN1>([&](auto a_) {
                constexpr int a = a_;
                constexpr int n = CH * IN1_D[a];
                for (int i = lane; i < n; i += 32)
                    cp_async_elem_fill((T*)dst + xs_off<a>() + i, row + IN1_OFF[a] + slice * n + i, be);
            });
        } else {
            for (int i = lane; i < X_DIM; i += 32) cp_async_elem_fill((T*)dst + i, row + i, be);
        }
    }
    // weights: path p of the slice is 32 consecutive values at W_OFF[p] + 32 slice, W_OFF[p] = 32 NSLICE p
    __device__ __forceinline__ void w_row(unsigned char* dst, const T* row, bool fill) const {
        if constexpr (!UNIT_W) {
            const int b16 = fill ? 0 : 16, be = fill ? 0 : ELEM;
            constexpr int PP = 32 / EPV;        // pieces per path and slice
            if (wv) {
#pragma unroll
                for (int i = 0; i < WI; ++i) {
                    const int q = lane + 32 * i;
                    if (32 * i + 32 <= WQ || q < WQ) {
                        if constexpr (FULL && N_SLICE > 1)
                            cp_async_16_hint(dst + 16 * q, row + slice * 32 + (lane / PP) * (32 * N_SLICE) + (lane % PP) * EPV +
                                                               i * (32 / PP) * (32 * N_SLICE), b16, stream);
                        else cp_async_16_hint(dst + 16 * q, row + q * EPV, b16, stream);
                    }
                }
            } else if constexpr (FULL && N_SLICE > 1) {
                for (int pth = 0; pth < N_INSTR; ++pth)
                    cp_async_elem_fill((T*)dst + 32 * pth + lane, row + (32 * N_SLICE) * pth + 32 * slice + lane, be);
            } else {
                for (int i = lane; i < W_NUMEL; i += 32) cp_async_elem_fill((T*)dst + i, row + i, be);
            }
        }
    }
    // A row of X values back to global memory: stored, or added.
    template <bool ADD>
    __device__ __forceinline__ void x_out(T* row, const T* src, bool vec) const {
        if constexpr (FULL && N_SLICE > 1) {
            if (vec) {
#pragma unroll
                for (int i = 0; i < XI; ++i) {
                    const int q = lane + 32 * i;
                    if (32 * i + 32 <= XQ || q < XQ) piece_out<ADD>(row + xo[i], src + q * EPV);
                }
            } else {
                sfor<0, N_IN1>([&](auto a_) {
                    constexpr int a = a_;
                    constexpr int n = CH * IN1_D[a];
                    for (int i = lane; i < n; i += 32) elem_out<ADD>(row + IN1_OFF[a] + slice * n + i, src[xs_off<a>() + i]);
                });
            }
        } else {
            if (vec) {
                for (int q = lane; q < XQ; q += 32) piece_out<ADD>(row + q * EPV, src + q * EPV);
            } else {
                for (int i = lane; i < X_DIM; i += 32) elem_out<ADD>(row + i, src[i]);
            }
        }
    }
    // A pair of one edge: the forward pass finds zeros in the place of the second one and adds them (a condition per path
    // and edge took more than the copies).  Elsewhere nothing is filled, and no copy asks for it: FP64 8x(0e+1o), 740 k edges,
    // deterministic forward 160 -> 154 us.
    static constexpr bool FILL = FORWARD && PK::N == 2;
    __device__ __forceinline__ void pair(const UvuParams& p, unsigned char* st, int e0, int row, int s0, int s1) const {
        using L = SliceStage;
        const bool two = s1 >= 0;
        if (lane == 0) *reinterpret_cast<int4*>(st + L::OFF_HDR) = make_int4(e0, row, s0, s1);
        auto y_rows = [&](const T* y, unsigned char* dst) {
            T* dy = reinterpret_cast<T*>(dst);
#pragma unroll
            for (int i = 0; i < (2 * Y_DIM + 31) / 32; ++i) {
                const int q = lane + 32 * i, h = q >= Y_DIM ? 1 : 0, j = q - h * Y_DIM;
                const bool fill = FILL && q >= Y_DIM && !two;
                if (q < (two || FILL ? 2 : 1) * Y_DIM) cp_async_elem_fill(dy + (PK::N == 2 ? 2 * j + h : q), fill ? y : y + q, fill ? 0 : ELEM);
            }
        };
        y_rows(p.Y + (long long)e0 * Y_DIM, st + L::OFF_Y);
        if constexpr (DBLC) y_rows(p.EY + (long long)e0 * Y_DIM, st + L::OFF_EY);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q == 0 || two || FILL) {
                const bool fill = q && !two;
                const long long s = q && two ? s1 : s0, e = e0 + (fill ? 0 : q);
                x_row(st + L::OFF_X + q * XSB, p.X + s * X_DIM, fill);
                w_row(st + L::OFF_W + q * WSB, p.W + e * W_NUMEL, fill);
                if constexpr (DBLC) {
                    x_row(st + L::OFF_EX + q * XSB, p.EX + s * X_DIM, fill);
                    w_row(st + L::OFF_EW + q * WSB, p.EW + e * W_NUMEL, fill);
                }
            }
        }
    }
};

// Pair of values of the two edges (FP32), or the value of edge h (FP64).
__device__ __forceinline__ V2 load_pair(const unsigned char* base, int stride_bytes, int el, int h) {
    const T* a = reinterpret_cast<const T*>(base) + el;
    if constexpr (PK::N == 2) return PK::make(a[0], a[stride_bytes / ELEM]);
    else return PK::make(a[h * (stride_bytes / ELEM)], (T)0);
}
template <class YA>
__device__ __forceinline__ void load_y(const unsigned char* base, int h, YA& y) {
    if constexpr (PK::N == 2) {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(base);
#pragma unroll
        for (int j = 0; j + 1 < Y_DIM; j += 2) {
            const ulonglong2 v = q[j / 2];
            y[j] = v.x;
            y[j + 1] = v.y;
        }
        if constexpr (Y_DIM % 2) y[Y_DIM - 1] = reinterpret_cast<const V2*>(base)[Y_DIM - 1];
    } else {
#pragma unroll
        for (int j = 0; j < Y_DIM; ++j) y[j] = reinterpret_cast<const V2*>(base)[h * Y_DIM + j];
    }
}


template <int O> __host__ __device__ constexpr int out_width() { return (FULL ? 32 : OUT_MUL[O]) * OUT_D[O]; }
template <int O> __host__ __device__ constexpr bool out_vec_ok() {
    return FULL || ((OUT_OFF[O] * ELEM) % 16 == 0 && (Z_DIM * ELEM) % 16 == 0 && (out_width<O>() * ELEM) % 16 == 0);
}

// ---------------------------------------------------------------- forward
//
// Bound by register reads: an FMA with an immediate reads two registers, one with three register operands three,
// and a scheduler's two banks deliver two a cycle.

// Second derivatives, gradient with respect to dZ: T(ex, y, w) + T(x, ey, w) + T(x, y, ew) of a pair, as one
// contraction: with r = w ex + ew x, t_ij = r_i y_j + (w x_i) ey_j and z_k += C_ijk t_ij.
template <class YA, class ZA>
__device__ __forceinline__ void slice_second_z(const unsigned char* st, int e, int lane, const YA& y, ZA& z) {
    using L = SliceStage;
    V2 ey[Y_DIM];
    load_y(st + L::OFF_EY, e, ey);
    sfor<0, N_IN1>([&](auto a_) {
        constexpr int a = a_;
        if constexpr (any_part_uses_in1(a)) {
            constexpr int D1 = IN1_D[a];
            const bool live = FULL || lane < IN1_MUL[a];
            V2 x[D1], ex[D1];
#pragma unroll
            for (int i = 0; i < D1; ++i) {
                x[i] = live ? load_pair(st + L::OFF_X, XSB, xs_off<a>() + lane * D1 + i, e) : PK::all((T)0);
                ex[i] = live ? load_pair(st + L::OFF_EX, XSB, xs_off<a>() + lane * D1 + i, e) : PK::all((T)0);
            }
            sfor<0, N_INSTR>([&](auto p_) {
                constexpr int P = p_;
                if constexpr (I_IN1[P] == a) {
                    constexpr int b = I_IN2[P], R = out_reg_off(I_OUT[P]);
                    const V2 w = live ? load_pair(st + L::OFF_W, WSB, ws_off<P>() + lane, e) : PK::all((T)0);
                    const V2 ew = live ? load_pair(st + L::OFF_EW, WSB, ws_off<P>() + lane, e) : PK::all((T)0);
                    V2 r[D1], wx[D1], t;
#pragma unroll
                    for (int i = 0; i < D1; ++i) {
                        r[i] = PK::fma(w, ex[i], PK::mul(ew, x[i]));
                        wx[i] = PK::mul(w, x[i]);
                    }
                    sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                        constexpr int n = n_;
                        constexpr int J = IN2_OFF[b] + CG_J[n];
                        if constexpr (cg_pair_first<P, n>()) t = PK::fma(r[CG_I[n]], y[J], PK::mul(wx[CG_I[n]], ey[J]));
                        T& zk = z[R + CG_K[n]];
                        zk = fma((T)CG_V[n], PK::get(t, 0), zk);
                        if constexpr (PK::N == 2) zk = fma((T)CG_V[n], PK::get(t, 1), zk);
                    });
                }
            });
        }
    });
}

// Where the weight of a path is applied that has its pair of inputs for itself: to the smallest of the three irreps.  On an
// input it takes products of two registers (an FMA of three costs half a clock more) and the coefficient FMAs go straight
// to the row.  With the zeros for a missing second edge: 32x(0e+1o+2e), 800 k edges, forward 281 -> 271 us; 128x(0e+1o+2e) x
// (0e..3o), 150 k edges, 313 -> 296; 128x(0e..3o), 1.2 M edges, 5.07 -> 4.86 ms.
enum class Place { IN1, IN2, OUT };
// FP64 with few sums: the coefficient FMAs of a path would follow one another on the same values of the row, at the FP64 FMA's
// latency.  740 k edges, weight on an input / on the output: 8x(0e+1o) with 0e+1o (8 sums) 163 / 153 us, to 0e..2e (13) 196 / 187, with
// 0e+1o+2e to 0e+1o (11) 210 / 196, but 8x(0e+1o+2e) with 0e (9, no two of a path on one sum) 153 / 157; 8x(1o+2e) with 0e+1o (17)
// 210 / 218, 8x(0e+2e) with 0e+2e (17) 241 / 243, 8x(0e+1o+2e) with 0e+1o (21) 247 / 249.  Rows of 32 channels: within 2 %.
constexpr bool FEW_SUMS = ELEM == 8 && ZPC_ALL < 16;
__host__ __device__ constexpr Place weight_place(int p) {
    const int d1 = IN1_D[I_IN1[p]], d2 = IN2_D[I_IN2[p]], d3 = OUT_D[I_OUT[p]];
    return d1 <= d2 && d1 <= d3 ? Place::IN1 : (d2 <= d3 ? Place::IN2 : Place::OUT);
}
__host__ __device__ constexpr bool same_coefficient(int p) {
    for (int n = CG_BEGIN[p]; n < CG_BEGIN[p + 1]; ++n)
        if (CG_V[n] != CG_V[CG_BEGIN[p]]) return false;
    return true;
}

// Output irrep O of a channel from its sums of products.
template <int O, class BA>
__device__ __forceinline__ void outer_contract(const BA& b, T (&v)[OUT_D[O]]) {
#pragma unroll
    for (int k = 0; k < OUT_D[O]; ++k) v[k] = (T)0;
    sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        if constexpr (I_OUT[P] == O) {
            sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                constexpr int n = n_;
                v[CG_K[n]] = fma((T)CG_V[n], b[CG_PR[n]], v[CG_K[n]]);
            });
        }
    });
}

template <int MODE>
__device__ void slice_forward(const UvuParams& p, unsigned char* smem, int warp, int lane) {
    using L = SliceStage;
    constexpr bool DET = MODE == MODE_DET;
    const int slice = warp % N_SLICE;
    const int walkers = (int)gridDim.x * (SL_WARPS / N_SLICE);
    PairWalker<DET> walk(p, walkers, (int)blockIdx.x * (SL_WARPS / N_SLICE) + warp / N_SLICE, lane);
    SliceCopies copies(p, slice, lane);
    unsigned char* stages = smem + (long long)warp * (SL_S * L::BYTES + SL_FLUSH);
    T* fbuf = reinterpret_cast<T*>(stages + SL_S * L::BYTES);
    const bool z_vec = p.flags & 8;

    // the receiver's row, or (OUTER) its sums of products
    constexpr int NZ = OUTER ? N_OUTER : ZPC_ALL;
    T z[NZ];
#pragma unroll
    for (int k = 0; k < NZ; ++k) z[k] = (T)0;

    auto flush = [&](int node) {
        T* zrow = p.Z + (long long)node * Z_DIM;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int o = o_;
            constexpr int D = OUT_D[o], R = out_reg_off(o);
            T* dst = zrow + OUT_OFF[o] + slice * out_width<o>();
            const bool live = FULL || lane < OUT_MUL[o];
            T v[D];
            if constexpr (OUTER) {
                outer_contract<o>(z, v);
            } else {
#pragma unroll
                for (int k = 0; k < D; ++k) v[k] = z[R + k];
            }
            if constexpr (D == 1) {
                if (live) {
                    if constexpr (DET) dst[lane] = v[0];
                    else red_add(dst + lane, v[0]);
                }
            } else {
                // [channel][component] rows: through shared memory, so that a warp's stores fill whole sectors
                if (live) {
#pragma unroll
                    for (int k = 0; k < D; ++k) fbuf[lane * D + k] = v[k];
                }
                __syncwarp();
                row_out<!DET>(dst, fbuf, out_width<o>(), z_vec && out_vec_ok<o>(), lane);
                __syncwarp();
            }
        });
#pragma unroll
        for (int k = 0; k < NZ; ++k) z[k] = (T)0;
    };

    bool more = true;
    int fill = 0, prev = -2, use = 0, ahead = 1 - SL_S;      // (the end of the walk is receiver -1)
    for (;;) {
        // stage the pair SL_S - 1 ahead
        {
            unsigned char* st = stages + fill * L::BYTES;
            fill = fill + 1 == SL_S ? 0 : fill + 1;
            if (more) {
                int e0, row, s0, s1, g0 = 0, g1 = 0;
                more = walk.next(e0, row, s0, s1, g0, g1);
                if (more) copies.pair(p, st, e0, row, s0, s1);
                else if (lane == 0) *reinterpret_cast<int4*>(st + L::OFF_HDR) = make_int4(0, -1, 0, 0);
                if constexpr (DET) {
                    // nodes without edges: zero rows, shared by the warps of a walker
                    if (more && (g0 < row || g1 > row + 1)) {
                        for (int node = g0; node < max(row, g1); node = node + 1 == row ? row + 1 : node + 1) {
                            if (node == row) continue;
                            T* zrow = p.Z + (long long)node * Z_DIM;
                            for (int i = slice * 32 + lane; i < Z_DIM; i += 32 * N_SLICE) zrow[i] = (T)0;
                        }
                    }
                }
            }
            cp_async_commit();
        }
        if (ahead < 0) {
            ++ahead;
            continue;
        }
        cp_async_wait<SL_S - 1>();
        __syncwarp();
        const unsigned char* st = stages + use * L::BYTES;
        use = use + 1 == SL_S ? 0 : use + 1;
        const int4 h = *reinterpret_cast<const int4*>(st + L::OFF_HDR);
        if (h.y != prev) {
            if (prev >= 0) flush(prev);
            prev = h.y;
            if (prev < 0) break;
        }
        const bool two = h.w >= 0;
        const unsigned char* sx = st + L::OFF_X;
        const unsigned char* sw = st + L::OFF_W;
#pragma unroll 1
        for (int e = 0; e < (PK::N == 2 || !two ? 1 : 2); ++e) {
            V2 y[Y_DIM];
            load_y(st + L::OFF_Y, e, y);
            if constexpr (DBLC) slice_second_z(st, e, lane, y, z);
            sfor<0, N_IN1>([&](auto a_) {
                constexpr int a = a_;
                if constexpr (any_part_uses_in1(a) && !DBLC) {
                    constexpr int D1 = IN1_D[a];
                    const bool live = FULL || lane < IN1_MUL[a];
                    V2 x[D1];
#pragma unroll
                    for (int i = 0; i < D1; ++i) x[i] = live ? load_pair(sx, XSB, xs_off<a>() + lane * D1 + i, e) : PK::all((T)0);
                    sfor<0, N_GROUPS>([&](auto g_) {
                        constexpr int g = g_;
                        if constexpr (GRP_A[g] == a && OUTER) {
                            sfor<GRP_PR[g], GRP_PR[g + 1]>([&](auto s_) {
                                constexpr int s = s_;
                                z[s] = fma(x[PR_I[s]], y[IN2_OFF[GRP_B[g]] + PR_J[s]], z[s]);
                            });
                        } else if constexpr (GRP_A[g] == a) {
                            constexpr int b = GRP_B[g], P0 = P_LIST[GRP_P[g]];
                            constexpr Place PL = UNIT_W || FEW_SUMS || GRP_P[g + 1] - GRP_P[g] > 1 ? Place::OUT : weight_place(P0);
                            if constexpr (PL == Place::OUT) {
                                V2 t[T_MAX], xy;
                                sfor<GRP_E[g], GRP_E[g + 1]>([&](auto n_) {
                                    constexpr int n = n_;
                                    if constexpr (E_NEW[n]) xy = PK::mul(x[E_I[n]], y[IN2_OFF[b] + E_J[n]]);
                                    if constexpr (E_FIRST[n]) t[E_T[n]] = PK::mul(xy, PK::all((T)E_V[n]));
                                    else t[E_T[n]] = PK::fma(xy, PK::all((T)E_V[n]), t[E_T[n]]);
                                });
                                sfor<GRP_P[g], GRP_P[g + 1]>([&](auto q_) {
                                    constexpr int P = P_LIST[q_], o = I_OUT[P], R = out_reg_off(o), TO = T_OFF[P];
                                    if constexpr (UNIT_W) {
#pragma unroll
                                        for (int k = 0; k < OUT_D[o]; ++k) {
                                            z[R + k] += PK::get(t[TO + k], 0);
                                            if constexpr (PK::N == 2) z[R + k] += PK::get(t[TO + k], 1);
                                        }
                                    } else {
                                        const V2 w = live ? load_pair(sw, WSB, ws_off<P>() + lane, e) : PK::all((T)0);
#pragma unroll
                                        for (int k = 0; k < OUT_D[o]; ++k) {
                                            z[R + k] = fma(PK::get(w, 0), PK::get(t[TO + k], 0), z[R + k]);
                                            if constexpr (PK::N == 2) z[R + k] = fma(PK::get(w, 1), PK::get(t[TO + k], 1), z[R + k]);
                                        }
                                    }
                                });
                            } else {
                                constexpr int R = out_reg_off(I_OUT[P0]);
                                const V2 w = live ? load_pair(sw, WSB, ws_off<P0>() + lane, e) : PK::all((T)0);
                                auto add = [&](auto n_, V2 u, V2 v) {        // z_k += u v of both edges
                                    constexpr int n = n_;
                                    T& zk = z[R + CG_K[n]];
                                    zk = fma(PK::get(u, 0), PK::get(v, 0), zk);
                                    if constexpr (PK::N == 2) zk = fma(PK::get(u, 1), PK::get(v, 1), zk);
                                };
                                constexpr int DW = PL == Place::IN1 ? IN1_D[GRP_A[g]] : IN2_D[b];
                                if constexpr (same_coefficient(P0) && DW == 1) {
                                    // a scalar input: its product with weight and coefficient scales the other one
                                    const V2 c = PK::mul(PK::mul(w, PL == Place::IN1 ? x[0] : y[IN2_OFF[b]]), PK::all((T)CG_V[CG_BEGIN[P0]]));
                                    sfor<CG_BEGIN[P0], CG_BEGIN[P0 + 1]>([&](auto n_) {
                                        constexpr int n = n_;
                                        add(n_, c, PL == Place::IN1 ? y[IN2_OFF[b] + CG_J[n]] : x[CG_I[n]]);
                                    });
                                } else {
                                    V2 v[DW], xy;
#pragma unroll
                                    for (int i = 0; i < DW; ++i) v[i] = PK::mul(w, PL == Place::IN1 ? x[i] : y[IN2_OFF[b] + i]);
                                    sfor<GRP_E[g], GRP_E[g + 1]>([&](auto n_) {
                                        constexpr int n = n_, k = E_T[n];
                                        if constexpr (E_NEW[n])
                                            xy = PL == Place::IN1 ? PK::mul(v[E_I[n]], y[IN2_OFF[b] + E_J[n]]) : PK::mul(x[E_I[n]], v[E_J[n]]);
                                        z[R + k] = fma((T)E_V[n], PK::get(xy, 0), z[R + k]);
                                        if constexpr (PK::N == 2) z[R + k] = fma((T)E_V[n], PK::get(xy, 1), z[R + k]);
                                    });
                                }
                            }
                        }
                    });
                }
            });
        }
        __syncwarp();       // every lane has read the stage: the next round refills it
    }
}


// ---------------------------------------------------------------- backward, receiver order
//
// Bound by issue: per edge and channel 2 three-register FMAs per (i, j) pair of every path plus the row-level sums.
// A channel's slice of dZ[receiver] stays in registers for a run of edges; P_ij = sum_k C_ijk dZ_k is formed once for
// both edges of a pair.  dX rows replace the staged X rows in shared memory and leave as 16-byte stores to the scratch
// row of the edge (deterministic: summed per sender afterwards) or as 16-byte additions to dX[sender] (atomic).

constexpr int DY_N = PK::N * Y_DIM;                                 // dY values of one step (two edges, or one in FP64)
constexpr int EPC = 16 / ELEM;                                      // elements per 16-byte piece
constexpr int DY_PITCH = DY_N > 32 ? (DY_N + 31) / 32 * 32 : imax(next_pow2(DY_N), 8);
constexpr int DY_COLS = DY_PITCH < 32 ? DY_PITCH : 32;              // values summed at a time, by 32 / DY_COLS lanes each
constexpr int DYB = 32 * DY_PITCH * ELEM;                           // transposition buffer of one warp
constexpr int DYG = N_SLICE > 1 ? 2 * N_SLICE * DY_PITCH * ELEM : 0;    // per walker: partial sums of the slices, two steps

// Element v of lane r in the transposition buffer: 16-byte pieces are permuted within a row so that neither the
// row-wise writes nor the column-wise reads meet on a bank.
__device__ __forceinline__ int dy_at(int r, int v) {
    constexpr int PIECES = DY_PITCH / EPC, M = PIECES < 8 ? PIECES - 1 : 7;
    const int c = v / EPC;
    return r * DY_PITCH + ((c & ~M) | ((c ^ (PIECES < 8 ? r * PIECES / 8 : r)) & M)) * EPC + v % EPC;
}

template <int MODE>
__device__ void slice_backward(const UvuParams& p, unsigned char* smem, int warp, int lane) {
    using L = SliceStage;
    constexpr bool DET = MODE == MODE_DET;
    constexpr int NE = PK::N;                   // edges computed together
    const int slice = warp % N_SLICE, grp = warp / N_SLICE;
    const int walkers = (int)gridDim.x * (SL_WARPS / N_SLICE);
    PairWalker<false> walk(p, walkers, (int)blockIdx.x * (SL_WARPS / N_SLICE) + grp, lane);
    SliceCopies copies(p, slice, lane);
    unsigned char* stages = smem + (long long)warp * (SL_S * L::BYTES + DYB);
    T* dyt = reinterpret_cast<T*>(stages + SL_S * L::BYTES);
    T* dyg = reinterpret_cast<T*>(smem + (long long)SL_WARPS * (SL_S * L::BYTES + DYB) + grp * DYG);
    const bool dx_vec = p.flags & 8;

    T gzc[CPL][OUTER ? N_OUTER : ZPC_ALL];      // the receiver's dZ, or (OUTER) its G
    auto& gz = gzc[0];
    bool more = true;
    int fill = 0, prev = -2, use = 0, ahead = 1 - SL_S, step = 0;
    for (;;) {
        {
            unsigned char* st = stages + fill * L::BYTES;
            fill = fill + 1 == SL_S ? 0 : fill + 1;
            if (more) {
                int e0, row, s0, s1, g0, g1;
                more = walk.next(e0, row, s0, s1, g0, g1);
                if (more) copies.pair(p, st, e0, row, s0, s1);
                else if (lane == 0) *reinterpret_cast<int4*>(st + L::OFF_HDR) = make_int4(0, -1, 0, 0);
            }
            cp_async_commit();
        }
        if (ahead < 0) {
            ++ahead;
            continue;
        }
        cp_async_wait<SL_S - 1>();
        __syncwarp();
        unsigned char* st = stages + use * L::BYTES;
        use = use + 1 == SL_S ? 0 : use + 1;
        const int4 h = *reinterpret_cast<const int4*>(st + L::OFF_HDR);
        if (h.y != prev) {
            prev = h.y;
            if (prev < 0) break;
            const T* zrow = p.dZ + (long long)prev * Z_DIM;
            if constexpr (OUTER) {
#pragma unroll
                for (int k = 0; k < CPL * N_OUTER; ++k) gzc[k / N_OUTER][k % N_OUTER] = (T)0;
            }
            sfor<0, N_OUT * CPL>([&](auto oc_) {
                constexpr int o = oc_ / CPL, c = oc_ % CPL;
                const bool live = FULL || lane < OUT_MUL[o];
                T v[OUT_D[o]];
#pragma unroll
                for (int k = 0; k < OUT_D[o]; ++k) v[k] = live ? __ldg(zrow + OUT_OFF[o] + (slice * CH + 32 * c + lane) * OUT_D[o] + k) : (T)0;
                if constexpr (OUTER) {
                    sfor<0, N_INSTR>([&](auto p_) {
                        constexpr int P = p_;
                        if constexpr (I_OUT[P] == o) {
                            sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                                constexpr int n = n_;
                                gzc[c][CG_PR[n]] = fma((T)CG_V[n], v[CG_K[n]], gzc[c][CG_PR[n]]);
                            });
                        }
                    });
                } else {
#pragma unroll
                    for (int k = 0; k < OUT_D[o]; ++k) gz[out_reg_off(o) + k] = v[k];
                }
            });
        }
        const bool two = h.w >= 0;
#pragma unroll 1
        for (int e = 0; e < (NE == 2 || !two ? 1 : 2); ++e) {
            T y[NE][Y_DIM], dy[NE][Y_DIM];
            {
                V2 yp[Y_DIM];
                load_y(st + L::OFF_Y, e, yp);
#pragma unroll
                for (int j = 0; j < Y_DIM; ++j) {
#pragma unroll
                    for (int q = 0; q < NE; ++q) {
                        y[q][j] = PK::get(yp[j], q);
                        dy[q][j] = (T)0;
                    }
                }
            }
            T* sx[NE];
            const T* sw[NE];
            T* dw[NE];
#pragma unroll
            for (int q = 0; q < NE; ++q) {
                sx[q] = reinterpret_cast<T*>(st + L::OFF_X + (e + q) * XSB);
                sw[q] = reinterpret_cast<const T*>(st + L::OFF_W + (e + q) * WSB);
                dw[q] = p.dW + (long long)(h.x + e + q) * W_NUMEL;
            }
            sfor<0, N_IN1 * CPL>([&](auto ac_) {
                constexpr int a = ac_ / CPL, c = ac_ % CPL, X0 = xs_off<a>() + 32 * c * IN1_D[a];
                constexpr int D1 = IN1_D[a];
                const bool live = FULL || lane < IN1_MUL[a];
                T x[NE][D1], dx[NE][D1], ex[DBLC ? NE : 1][D1];
#pragma unroll
                for (int q = 0; q < NE; ++q)
#pragma unroll
                    for (int i = 0; i < D1; ++i) {
                        x[q][i] = live ? sx[q][X0 + lane * D1 + i] : (T)0;
                        dx[q][i] = (T)0;
                        if constexpr (DBLC) ex[q][i] = live ? sx[q][(L::OFF_EX - L::OFF_X) / ELEM + xs_off<a>() + lane * D1 + i] : (T)0;
                    }
                if constexpr (OUTER) {
                    sfor<0, N_GROUPS>([&](auto g_) {
                        constexpr int g = g_;
                        if constexpr (GRP_A[g] == a) {
                            sfor<GRP_PR[g], GRP_PR[g + 1]>([&](auto s_) {
                                constexpr int s = s_, i = PR_I[s], j = IN2_OFF[GRP_B[g]] + PR_J[s];
#pragma unroll
                                for (int q = 0; q < NE; ++q) {
                                    dx[q][i] = fma(y[q][j], gzc[c][s], dx[q][i]);
                                    dy[q][j] = fma(x[q][i], gzc[c][s], dy[q][j]);
                                }
                            });
                        }
                    });
                }
                sfor<0, N_INSTR>([&](auto p_) {
                    constexpr int P = p_;
                    if constexpr (OUTER) {
                    } else if constexpr (I_IN1[P] == a && DBLC) {
                        // gx = w A(ey) + ew A(y), gw = <ex, A(y)> + <x, A(ey)>, gy = B(w ex + ew x) with
                        // A_i(v) = sum_j v_j P_ij, B_j(v) = sum_i v_i P_ij; the same with the inputs exchanged where the
                        // second one is smaller (six FMAs per value of the smaller input)
                        constexpr int b = I_IN2[P], D2 = IN2_D[b], R = out_reg_off(I_OUT[P]);
                        constexpr bool W1 = D1 <= D2;
                        constexpr int DM = W1 ? D1 : D2;
                        T w[NE], ew[NE], r[NE][DM], ay[NE][DM], ae[NE][DM], ey[NE][D2], pij = (T)0;
#pragma unroll
                        for (int q = 0; q < NE; ++q) {
                            w[q] = live ? sw[q][ws_off<P>() + lane] : (T)0;
                            ew[q] = live ? sw[q][(L::OFF_EW - L::OFF_W) / ELEM + ws_off<P>() + lane] : (T)0;
                            const T* sey = reinterpret_cast<const T*>(st + L::OFF_EY) + (NE == 2 ? q : e * Y_DIM);
#pragma unroll
                            for (int j = 0; j < D2; ++j) ey[q][j] = sey[(IN2_OFF[b] + j) * NE];
#pragma unroll
                            for (int i = 0; i < DM; ++i) {
                                r[q][i] = W1 ? fma(w[q], ex[q][W1 ? i : 0], ew[q] * x[q][W1 ? i : 0])
                                             : fma(w[q], ey[q][W1 ? 0 : i], ew[q] * y[q][IN2_OFF[b] + (W1 ? 0 : i)]);
                                ay[q][i] = ae[q][i] = (T)0;
                            }
                        }
                        sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                            constexpr int n = n_, i = CG_I[n], j = CG_J[n], m = W1 ? i : j;
                            if constexpr (cg_pair_first<P, n>()) pij = (T)CG_V[n] * gz[R + CG_K[n]];
                            else pij = fma((T)CG_V[n], gz[R + CG_K[n]], pij);
                            if constexpr (cg_pair_last<P, n>()) {
#pragma unroll
                                for (int q = 0; q < NE; ++q) {
                                    ay[q][m] = fma(W1 ? y[q][IN2_OFF[b] + j] : x[q][i], pij, ay[q][m]);
                                    ae[q][m] = fma(W1 ? ey[q][j] : ex[q][i], pij, ae[q][m]);
                                    T& d = W1 ? dy[q][IN2_OFF[b] + j] : dx[q][i];
                                    d = fma(r[q][m], pij, d);
                                }
                            }
                        });
#pragma unroll
                        for (int q = 0; q < NE; ++q) {
                            T gw = (T)0;
#pragma unroll
                            for (int i = 0; i < DM; ++i) {
                                gw = fma(W1 ? ex[q][W1 ? i : 0] : ey[q][W1 ? 0 : i], ay[q][i], gw);
                                gw = fma(W1 ? x[q][W1 ? i : 0] : y[q][IN2_OFF[b] + (W1 ? 0 : i)], ae[q][i], gw);
                                T& d = W1 ? dx[q][W1 ? i : 0] : dy[q][IN2_OFF[b] + (W1 ? 0 : i)];
                                d = fma(w[q], ae[q][i], d);
                                d = fma(ew[q], ay[q][i], d);
                            }
                            if (live && (q == 0 || two)) __stcs(dw[q] + W_OFF[P] + slice * 32 + lane, gw);
                        }
                    } else if constexpr (I_IN1[P] == a) {
                        constexpr int b = I_IN2[P], D2 = IN2_D[b], R = out_reg_off(I_OUT[P]);
                        // The weight goes to the smaller input: with w x in dY's sums, sum_j y_j P_ij gives dW and, times w,
                        // dX (or the same with the inputs exchanged).  The kernel is bound by register reads; 128x(0e+1o+2e) x
                        // (0e..3o), 150 k edges: 446 -> 414 FMAs per edge and 32 channels, 619 -> 596 us.
                        constexpr bool W1 = D1 <= D2;
                        T wv[NE][W1 ? D1 : D2], sv[NE][W1 ? D1 : D2], w[NE], pij = (T)0;
                        if constexpr (!UNIT_W) {
#pragma unroll
                            for (int q = 0; q < NE; ++q) {
                                w[q] = live ? sw[q][ws_off<P>() + lane] : (T)0;
#pragma unroll
                                for (int i = 0; i < (W1 ? D1 : D2); ++i) {
                                    wv[q][i] = w[q] * (W1 ? x[q][i] : y[q][IN2_OFF[b] + i]);
                                    sv[q][i] = (T)0;
                                }
                            }
                        }
                        sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                            constexpr int n = n_, i = CG_I[n], j = CG_J[n];
                            if constexpr (cg_pair_first<P, n>()) pij = (T)CG_V[n] * gz[R + CG_K[n]];
                            else pij = fma((T)CG_V[n], gz[R + CG_K[n]], pij);
                            if constexpr (cg_pair_last<P, n>()) {
#pragma unroll
                                for (int q = 0; q < NE; ++q) {
                                    T& ai = UNIT_W || !W1 ? dx[q][i] : sv[q][W1 ? i : 0];
                                    T& bj = UNIT_W || W1 ? dy[q][IN2_OFF[b] + j] : sv[q][W1 ? 0 : j];
                                    ai = fma(UNIT_W || W1 ? y[q][IN2_OFF[b] + j] : wv[q][W1 ? 0 : j], pij, ai);
                                    bj = fma(UNIT_W || !W1 ? x[q][i] : wv[q][W1 ? i : 0], pij, bj);
                                }
                            }
                        });
                        if constexpr (!UNIT_W) {
#pragma unroll
                            for (int q = 0; q < NE; ++q) {
                                T tw = (T)0;
#pragma unroll
                                for (int i = 0; i < (W1 ? D1 : D2); ++i) {
                                    tw = fma(W1 ? x[q][i] : y[q][IN2_OFF[b] + i], sv[q][i], tw);
                                    T& d = W1 ? dx[q][i] : dy[q][IN2_OFF[b] + i];
                                    d = fma(w[q], sv[q][i], d);
                                }
                                if (live && (q == 0 || two)) __stcs(dw[q] + W_OFF[P] + slice * 32 + lane, tw);
                            }
                        }
                    }
                });
                if (live) {
#pragma unroll
                    for (int q = 0; q < NE; ++q)
#pragma unroll
                        for (int i = 0; i < D1; ++i) sx[q][X0 + lane * D1 + i] = dx[q][i];
                }
            });
            // dY: transpose through shared memory, lane v then owns value v (edge-major) of all 32 channels
#pragma unroll
            for (int v = 0; v < DY_PITCH; v += EPC) {
                if (v < DY_N) {
                    T t[EPC];
#pragma unroll
                    for (int i = 0; i < EPC; ++i) {
                        const int vi = v + i;
                        t[i] = vi < DY_N ? dy[vi / Y_DIM][vi % Y_DIM] : (T)0;
                    }
                    if constexpr (ELEM == 4) *reinterpret_cast<float4*>(dyt + dy_at(lane, v)) = make_float4(t[0], t[1], t[2], t[3]);
                    else *reinterpret_cast<double2*>(dyt + dy_at(lane, v)) = make_double2(t[0], t[1]);
                }
            }
            __syncwarp();       // (also: the dX rows are complete)
            {
                const int n_dy = (NE == 2 && two ? 2 : 1) * Y_DIM;
                T* dyrow = p.dY + (long long)(h.x + e) * Y_DIM;
                T* mine = dyg + ((step & 1) * N_SLICE + slice) * DY_PITCH;
#pragma unroll
                for (int v0 = 0; v0 < DY_PITCH; v0 += DY_COLS) {
                    constexpr int ROWS = DY_COLS;       // rows that a lane adds up: 32 / (32 / DY_COLS)
                    const int v = v0 + lane % DY_COLS, r0 = lane / DY_COLS * ROWS;
                    T s4[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) s4[r & 3] += dyt[dy_at(r0 + r, v)];
                    T s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
#pragma unroll
                    for (int off = DY_COLS; off < 32; off *= 2) s += __shfl_xor_sync(0xffffffffu, s, off);
                    if (lane < DY_COLS) {
                        if constexpr (N_SLICE == 1) {
                            if (v < n_dy) dyrow[v] = s;
                        } else {
                            mine[v] = s;
                        }
                    }
                }
                if constexpr (N_SLICE > 1) {
                    group_sync(1 + grp, 32 * N_SLICE);
                    if (step % N_SLICE == slice) {
                        const T* part = dyg + (step & 1) * N_SLICE * DY_PITCH;
                        for (int v = lane; v < n_dy; v += 32) {
                            T s = part[v];
#pragma unroll
                            for (int q = 1; q < N_SLICE; ++q) s += part[q * DY_PITCH + v];
                            dyrow[v] = s;
                        }
                    }
                }
                ++step;
            }
            if constexpr (NE == 1) __syncwarp();    // the transposition buffer has been read
        }
        // dX rows of the two edges
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q == 0 || two) {
                T* row = DET ? p.ws + (long long)(h.x + q) * (XB / ELEM) : p.dX + (long long)(q ? h.w : h.z) * X_DIM;
                copies.x_out<!DET>(row, reinterpret_cast<const T*>(st + L::OFF_X + q * XSB), dx_vec);
            }
        }
        __syncwarp();       // every lane has read the stage: the next round refills it
    }
}

}  // namespace oeq

extern "C" __global__ void __launch_bounds__(32 * oeq::SL_WARPS, oeqd::MIN_CTAS) oeq_uvu_kernel(const oeq::UvuParams p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#if OEQ_KERNEL == OEQ_K_SLICE_FWD_DET
    oeq::slice_forward<oeq::MODE_DET>(p, smem_raw, warp, lane);
#elif OEQ_KERNEL == OEQ_K_SLICE_FWD_ATOMIC
    oeq::slice_forward<oeq::MODE_ATOMIC>(p, smem_raw, warp, lane);
#elif OEQ_KERNEL == OEQ_K_SLICE_DBL_Z_DET
    oeq::slice_forward<oeq::MODE_DET>(p, smem_raw, warp, lane);
#elif OEQ_KERNEL == OEQ_K_SLICE_DBL_Z_ATOMIC
    oeq::slice_forward<oeq::MODE_ATOMIC>(p, smem_raw, warp, lane);
#elif OEQ_KERNEL == OEQ_K_SLICE_BWD_DET || OEQ_KERNEL == OEQ_K_SLICE_DBL_G_DET
    oeq::slice_backward<oeq::MODE_DET>(p, smem_raw, warp, lane);
#elif OEQ_KERNEL == OEQ_K_SLICE_BWD_ATOMIC || OEQ_KERNEL == OEQ_K_SLICE_DBL_G_ATOMIC
    oeq::slice_backward<oeq::MODE_ATOMIC>(p, smem_raw, warp, lane);
#else
#error "OEQ_KERNEL must select one of the slice kernels"
#endif
}
