// "uvw" tensor product in FP64 with shared weights and second-input multiplicity 1, as register-tiled GEMMs on the
// FP64 FMA pipe (64 FMA per clock and SM: the bound).
//
//   product:  Z[b,o,w,k] = sum_{paths p -> o} sum_u W_p[u,w] T_p[b,u,k]   a CTA owns 64 (row, component) pairs x 64 w of
//             one output irrep and walks the paths in chunks of 32 u.  Also dT = W dZ of the backward pass (UNIT_Y: the
//             operand is dZ itself, weights transposed, the paths that share dZ joined in one output block).
//   dW:       dW_p[u,w] = sum_{b,k} T_p[b,u,k] dZ[b,o,w,k]                a CTA owns 64 u x 64 w of one path and a share
//             of the rows; the shares are added afterwards in a fixed order.
//
// T_p[b,u,k] = sum_ij C_p[i,j,k] x[b,u,i] y[b,j] is formed in shared memory where it is used.  Eight warps, a 4 x 4
// register tile per thread: a k step reads 4 shared-memory wavefronts per warp for 32 cycles of FMAs.  The chunk ahead
// is formed in the other buffer, so that its global loads overlap other warps' arithmetic.  The tiled kernel of
// uvw_kernels.cuh read weights from global memory, a different row per lane, and two operands per FMA from shared memory.
// Measured, 64x(0e+1o+2e) x (0e+1o+2e): 43 593 rows forward 1.81 ms and 9 925 rows forward + backward 3.18 ms before,
// 0.89 and 0.77 ms with these kernels.
#pragma once
#include "oeq_common.cuh"

#define OEQ_K_UVW_GEMM 14
#define OEQ_K_UVW_GEMM_DW 15

namespace oeq {
using namespace oeqd;

struct UvwGemmParams {
    const T* X;
    const T* Y;
    const T* W;
    const T* dZ;
    T* Z;               // product
    T* ws;              // dW: [shares][W_NUMEL]
    long long batch;
    int shares;
};

constexpr int GT = 64, GK = 32;                 // tile edge, depth of a chunk
constexpr int G_THREADS = 256;
constexpr int G_PITCH = GT + 2;                 // 16-byte aligned rows; columns written at this stride meet two to a bank
constexpr int G_BUF = GK * G_PITCH;

__host__ __device__ constexpr int g_rows(int o) { return GT / OUT_D[o]; }          // product: batch rows of a tile
__host__ __device__ constexpr int g_wtiles(int o) { return (OUT_MUL[o] + GT - 1) / GT; }

template <int P, class XA, class YA, class TA>
__device__ __forceinline__ void g_form(const XA& x, const YA& y, TA& t) {
#pragma unroll
    for (int k = 0; k < OUT_D[I_OUT[P]]; ++k) t[k] = (T)0;
    if constexpr (UNIT_Y) {
#pragma unroll
        for (int k = 0; k < OUT_D[I_OUT[P]]; ++k) t[k] = x[k];
    } else {
        T xy = (T)0;
        sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
            constexpr int N = n_;
            if constexpr (N == CG_BEGIN[P] || CG_I[N] != CG_I[N - 1] || CG_J[N] != CG_J[N - 1]) xy = x[CG_I[N]] * y[CG_J[N]];
            t[CG_K[N]] = fma(xy, (T)CG_V[N], t[CG_K[N]]);
        });
    }
}

// T of path P, channel u and batch row `row` (zeros outside).
template <int P, class TA>
__device__ __forceinline__ void g_t(const UvwGemmParams& p, long long row, int u, bool live, TA& t) {
    constexpr int a = I_IN1[P], b = I_IN2[P], D1 = IN1_D[a], D2 = IN2_D[b];
    T x[D1], y[D2];
    const T* xr = p.X + row * X_DIM + IN1_OFF[a] + u * D1;
#pragma unroll
    for (int i = 0; i < D1; ++i) x[i] = live ? __ldg(xr + i) : (T)0;
    if constexpr (!UNIT_Y) {
        const T* yr = p.Y + row * Y_DIM + IN2_OFF[b];
#pragma unroll
        for (int j = 0; j < D2; ++j) y[j] = live ? __ldg(yr + j) : (T)0;
    }
    g_form<P>(x, y, t);
}

// A warp owns 16 x 32 of the tile (lanes 4 x 8), a thread two pairs of rows and two pairs of columns: every 16-byte read
// of a k step is one wavefront.
__device__ __forceinline__ int g_row(int tid, int i) { return (tid >> 6) * 16 + ((tid >> 3) & 3) * 2 + (i & 1) + (i >> 1) * 8; }
__device__ __forceinline__ int g_col(int tid, int j) { return ((tid >> 5) & 1) * 32 + (tid & 7) * 2 + (j & 1) + (j >> 1) * 16; }

// acc[i][j] += sum over the chunk of a[.][g_row(i)] b[.][g_col(j)]
__device__ __forceinline__ void g_chunk(const T* a, const T* b, int depth, T (&acc)[4][4]) {
    const int tid = threadIdx.x;
    a += g_row(tid, 0);
    b += g_col(tid, 0);
#pragma unroll 4
    for (int k = 0; k < depth; ++k) {
        const double2 a0 = *reinterpret_cast<const double2*>(a + k * G_PITCH), a1 = *reinterpret_cast<const double2*>(a + k * G_PITCH + 8);
        const double2 b0 = *reinterpret_cast<const double2*>(b + k * G_PITCH), b1 = *reinterpret_cast<const double2*>(b + k * G_PITCH + 16);
        const T av[4] = {a0.x, a0.y, a1.x, a1.y}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
}

// Weight of path P, input channel u, output channel w.
template <int P>
__device__ __forceinline__ T g_weight(const T* W, int u, int w) {
    constexpr int MU = IN1_MUL[I_IN1[P]], MW = OUT_MUL[I_OUT[P]];
    if (u >= MU || w >= MW) return (T)0;
    if constexpr (TRANSPOSED_W) {
        T v = (T)0;
        sfor<SUB_BEGIN[P], SUB_BEGIN[P + 1]>([&](auto q_) {
            constexpr int q = q_;
            if (w >= SUB_START[q] && w < SUB_START[q] + SUB_MUL[q])
                v = __ldg(W + SUB_WOFF[q] + weight_offset_v1(SUB_MUL[q], MU, w - SUB_START[q], u));
        });
        return v;
    } else {
        return __ldg(W + W_OFF[P] + weight_offset_v1(MU, MW, u, w));
    }
}

// ---------------------------------------------------------------- product

template <int O>
__device__ void g_product(const UvwGemmParams& p, T* smem, long long tile, int w0) {
    constexpr int D3 = OUT_D[O], RT = g_rows(O), MW = OUT_MUL[O];
    const int tid = threadIdx.x;
    const long long b0 = tile * RT;
    if (b0 >= p.batch) return;
    const int rows = (int)(p.batch - b0 < RT ? p.batch - b0 : RT);
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = (T)0;
    int buf = 0;
    sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        if constexpr (I_OUT[P] == O) {
            constexpr int MU = IN1_MUL[I_IN1[P]];
#pragma unroll 1
            for (int u0 = 0; u0 < MU; u0 += GK, buf ^= 1) {
                T* as = smem + buf * 2 * G_BUF;
                T* bs = as + G_BUF;
                // (a warp forms chunk n while others still read chunk n - 1, never n - 2: everyone has passed n - 1's barrier)
                for (int item = tid; item < GK * RT; item += G_THREADS) {
                    const int ul = item % GK, r = item / GK;
                    T t[D3];
                    g_t<P>(p, b0 + (r < rows ? r : 0), u0 + ul, r < rows && u0 + ul < MU, t);
#pragma unroll
                    for (int k = 0; k < D3; ++k) as[ul * G_PITCH + r * D3 + k] = t[k];
                }
#pragma unroll 4
                for (int item = tid; item < GK * GT; item += G_THREADS) {
                    const int ul = TRANSPOSED_W ? item % GK : item / GT, w = TRANSPOSED_W ? item / GK : item % GT;
                    bs[ul * G_PITCH + w] = g_weight<P>(p.W, u0 + ul, w0 + w);
                }
                __syncthreads();
                g_chunk(as, bs, MU - u0 < GK ? MU - u0 : GK, acc);
            }
        }
    });
    // [row][w][k] through shared memory, so that rows are written contiguously
    __syncthreads();
    const int live = (MW - w0 < GT ? MW - w0 : GT) * D3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = g_row(tid, i), r = m / D3, k = m - r * D3;
        if (r < RT) {
#pragma unroll
            for (int j = 0; j < 4; ++j) smem[r * (GT * D3) + g_col(tid, j) * D3 + k] = acc[i][j];
        }
    }
    __syncthreads();
    for (int e = tid; e < rows * GT * D3; e += G_THREADS) {
        const int r = e / (GT * D3), c = e - r * (GT * D3);
        if (c < live) p.Z[(b0 + r) * Z_DIM + OUT_OFF[O] + w0 * D3 + c] = smem[e];
    }
}

// ---------------------------------------------------------------- weight gradient

template <int P>
__device__ void g_dw(const UvwGemmParams& p, T* smem, int share, int u0, int w0) {
    constexpr int o = I_OUT[P], D3 = OUT_D[o], MU = IN1_MUL[I_IN1[P]], MW = OUT_MUL[o], RC = GK / D3;
    const int tid = threadIdx.x;
    const long long lo = p.batch * share / p.shares, hi = p.batch * (share + 1) / p.shares;
    const int wn = (MW - w0 < GT ? MW - w0 : GT) * D3;
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = (T)0;
    int buf = 0;
#pragma unroll 1
    for (long long b0 = lo; b0 < hi; b0 += RC, buf ^= 1) {
        T* as = smem + buf * 2 * G_BUF;
        T* bs = as + G_BUF;
        const int rows = (int)(hi - b0 < RC ? hi - b0 : RC);
        for (int item = tid; item < rows * GT; item += G_THREADS) {
            const int u = item % GT, r = item / GT;
            T t[D3];
            g_t<P>(p, b0 + r, u0 + u, u0 + u < MU, t);
#pragma unroll
            for (int k = 0; k < D3; ++k) as[(r * D3 + k) * G_PITCH + u] = t[k];
        }
        for (int item = tid; item < rows * GT * D3; item += G_THREADS) {
            const int r = item / (GT * D3), c = item - r * (GT * D3);
            bs[(r * D3 + c % D3) * G_PITCH + c / D3] = c < wn ? __ldg(p.dZ + (b0 + r) * Z_DIM + OUT_OFF[o] + w0 * D3 + c) : (T)0;
        }
        __syncthreads();
        g_chunk(as, bs, rows * D3, acc);
    }
    T* out = p.ws + (long long)share * W_NUMEL + W_OFF[P];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int u = u0 + g_row(tid, i), w = w0 + g_col(tid, j);
            if (u < MU && w < MW) out[weight_offset_v1(MU, MW, u, w)] = acc[i][j];
        }
}

}  // namespace oeq

// Grid: x = row tile (or share of the rows), y = tile of 64 output channels over all output irreps (or of 64 u x 64 w
// over all paths).
extern "C" __global__ void __launch_bounds__(oeq::G_THREADS, 2) oeq_uvw_gemm_kernel(const oeq::UvwGemmParams p) {
    using namespace oeqd;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(smem_raw);
    int y = blockIdx.y;
#if OEQ_KERNEL == OEQ_K_UVW_GEMM
    oeq::sfor<0, N_OUT>([&](auto o_) {
        constexpr int O = o_, N = oeq::g_wtiles(O);
        if (y >= 0 && y < N) oeq::g_product<O>(p, smem, blockIdx.x, y * oeq::GT);
        y -= N;
    });
#elif OEQ_KERNEL == OEQ_K_UVW_GEMM_DW
    oeq::sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_, NW = oeq::g_wtiles(I_OUT[P]), N = (IN1_MUL[I_IN1[P]] + oeq::GT - 1) / oeq::GT * NW;
        if (y >= 0 && y < N) oeq::g_dw<P>(p, smem, blockIdx.x, y / NW * oeq::GT, y % NW * oeq::GT);
        y -= N;
    });
#else
#error "OEQ_KERNEL must select one of the GEMM kernels"
#endif
}

// Fixed-order sum of the partial weight gradients.
extern "C" __global__ void __launch_bounds__(256) oeq_reduce_partials(const oeqd::T* ws, oeqd::T* out, int n, long long groups) {
    oeq::reduce_partials(ws, out, n, groups);
}
