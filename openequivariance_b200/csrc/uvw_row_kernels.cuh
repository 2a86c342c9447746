// "uvw" tensor product with weights of its own for every row: one row per CTA.
//
// Every weight is used once, so the rate of the weight array is the floor (a row of 10x1o+10x1e+48x0e+48x0o reads
// 27.7 KB of weights against 1.3 KB of everything else).  The tiled kernel of uvw_kernels.cuh takes 16 rows per CTA,
// which leaves a batch of two thousand rows on 126 of 148 SMs and reads each row's weights a few at a time.  Here a
// CTA of eight warps takes a row, lanes run along the output channels (coalesced weights), eight weights of
// consecutive input channels are in flight per lane, and several rows share an SM.
//   forward:  a warp owns 32 output channels and adds up W[u,v,w] T[u,v,k] over all paths into them.
//   backward: a warp owns eight input channels of a path: dW[u,v,w] = sum_k T[u,v,k] dZ[w,k] leaves at once, and
//             dT[u,v,k] = sum_w W[u,v,w] dZ[w,k] is reduced over the lanes by recursive halving (fixed order);
//             dX and dY follow from dT.
// Measured, 2011 rows of the irreps above with a 1x0e+1x1o second input, FP32: forward 94 -> 24 us, backward 115 -> 33 us
// (the weights alone take 8.5 and 17 us at the copy bandwidth).
// What bounds it now is latency and the barriers of a row's phases: at 5 000 rows DRAM runs at 34 % of its rate, 39 and 50 % of
// the cycles issue.  Rows with few weights keep the tiled kernel beyond some rows per SM (uvw_row_limit).
#pragma once
#include "uvw_kernels.cuh"

#define OEQ_K_UVW_ROW_FWD 12
#define OEQ_K_UVW_ROW_BWD 13

namespace oeq {

constexpr int RW = ROW_WARPS, RT_THREADS = 32 * ROW_WARPS;
__host__ __device__ constexpr int t_offset(int p) {
    int n = 0;
    for (int q = 0; q < p; ++q) n += IN1_MUL[I_IN1[q]] * IN2_MUL[I_IN2[q]] * OUT_D[I_OUT[q]];
    return n;
}
constexpr int T_ALL = t_offset(N_INSTR);
constexpr int UG = 8;       // input channels of a backward step

__host__ __device__ constexpr int r4(int n) { return (n + 3) / 4 * 4; }
struct RowSmem {
    T *xs, *ys, *zs, *t, *dt, *gy;
    __device__ explicit RowSmem(unsigned char* raw) {
        xs = reinterpret_cast<T*>(raw);
        ys = xs + r4(X_DIM);
        zs = ys + r4(Y_DIM);
        t = zs + r4(Z_DIM);
        dt = t + r4(T_ALL);         // backward only
        gy = dt + r4(T_ALL);        // [RW][Y_DIM]
    }
};

// T of the row, [path][u][v][k].
__device__ __forceinline__ void row_t(const RowSmem& s, int tid) {
    sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        constexpr int a = I_IN1[P], b = I_IN2[P], o = I_OUT[P];
        constexpr int D1 = IN1_D[a], D2 = IN2_D[b], D3 = OUT_D[o], MV = IN2_MUL[b];
        // (paths start at different threads, so that short ones do not all land on the first warp)
        for (int uv = (tid + 32 * P) % RT_THREADS; uv < IN1_MUL[a] * MV; uv += RT_THREADS) {
            const int u = uv / MV, v = uv % MV;
            T x[D1], y[D2], t[D3];
#pragma unroll
            for (int i = 0; i < D1; ++i) x[i] = s.xs[IN1_OFF[a] + u * D1 + i];
#pragma unroll
            for (int j = 0; j < D2; ++j) y[j] = s.ys[IN2_OFF[b] + v * D2 + j];
#pragma unroll
            for (int k = 0; k < D3; ++k) t[k] = (T)0;
            uvw_cg_forward<P>(x, y, t);
#pragma unroll
            for (int k = 0; k < D3; ++k) s.t[t_offset(P) + uv * D3 + k] = t[k];
        }
    });
}

// Weights of path P, input chunk (uc, vc), output chunk wc: a contiguous block [v][u][w].
template <int P>
__device__ __forceinline__ int row_block(int uc, int vc, int wc, int ulen, int vlen) {
    constexpr int MV = IN2_MUL[I_IN2[P]], MW = OUT_MUL[I_OUT[P]];
    return W_OFF[P] + (uc * 32) * MV * MW + ulen * ((vc * 32) * MW + vlen * (wc * 32));
}

__device__ void uvw_row_forward(const UvwParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const RowSmem s(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long row = blockIdx.x; row < p.batch; row += gridDim.x) {
        for (int i = tid; i < X_DIM; i += RT_THREADS) s.xs[i] = p.X[row * X_DIM + i];
        for (int i = tid; i < Y_DIM; i += RT_THREADS) s.ys[i] = p.Y[row * Y_DIM + i];
        __syncthreads();
        row_t(s, tid);
        __syncthreads();
        const T* wrow = p.W + row * (long long)W_NUMEL;
        T* zrow = p.Z + row * (long long)Z_DIM;
        int tile = 0;       // 32 output channels of an output irrep
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int o = o_;
            constexpr int D3 = OUT_D[o], MW = OUT_MUL[o], WCS = (MW + 31) / 32;
            for (int wc = 0; wc < WCS; ++wc, ++tile) {
                if (tile % RW != warp) continue;
                const int wlen = MW - wc * 32 < 32 ? MW - wc * 32 : 32;
                const bool live = lane < wlen;
                T acc[D3];
#pragma unroll
                for (int k = 0; k < D3; ++k) acc[k] = (T)0;
                sfor<0, N_INSTR>([&](auto p_) {
                    constexpr int P = p_;
                    if constexpr (I_OUT[P] == o) {
                        constexpr int MU = IN1_MUL[I_IN1[P]], MV = IN2_MUL[I_IN2[P]];
                        for (int uc = 0; uc < (MU + 31) / 32; ++uc) {
                            const int ulen = MU - uc * 32 < 32 ? MU - uc * 32 : 32;
                            for (int vc = 0; vc < (MV + 31) / 32; ++vc) {
                                const int vlen = MV - vc * 32 < 32 ? MV - vc * 32 : 32;
                                const T* w = wrow + row_block<P>(uc, vc, wc, ulen, vlen) + lane;
                                for (int vl = 0; vl < vlen; ++vl) {
                                    const T* t = s.t + t_offset(P) + (uc * 32 * MV + vc * 32 + vl) * D3;
                                    const T* wv = w + vl * ulen * wlen;
#pragma unroll 8
                                    for (int ul = 0; ul < ulen; ++ul) {
                                        const T q = live ? __ldcs(wv + ul * wlen) : (T)0;
#pragma unroll
                                        for (int k = 0; k < D3; ++k) acc[k] = fma(q, t[ul * MV * D3 + k], acc[k]);
                                    }
                                }
                            }
                        }
                    }
                });
                if (live) {
#pragma unroll
                    for (int k = 0; k < D3; ++k) zrow[OUT_OFF[o] + (wc * 32 + lane) * D3 + k] = acc[k];
                }
            }
        });
        __syncthreads();        // T and the inputs are free for the next row
    }
}

// Sum each of v[0..8) over the 32 lanes in a fixed order; lane L ends with the total of value L >> 2 in v[0].
template <class VA>
__device__ __forceinline__ void warp_reduce_8(VA& v, int lane) {
#pragma unroll
    for (int off = 16, half = UG / 2; off > 0; off >>= 1, half >>= 1) {
        if (half > 0) {
            const bool upper = (lane & off) != 0;
#pragma unroll
            for (int m = 0; m < UG / 2; ++m)
                if (m < half) {
                    const T send = upper ? v[m] : v[m + half], keep = upper ? v[m + half] : v[m];
                    v[m] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        }
    }
}

__device__ void uvw_row_backward(const UvwParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const RowSmem s(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long row = blockIdx.x; row < p.batch; row += gridDim.x) {
        for (int i = tid; i < X_DIM; i += RT_THREADS) s.xs[i] = p.X[row * X_DIM + i];
        for (int i = tid; i < Y_DIM; i += RT_THREADS) s.ys[i] = p.Y[row * Y_DIM + i];
        for (int i = tid; i < Z_DIM; i += RT_THREADS) s.zs[i] = p.dZ[row * Z_DIM + i];
        for (int i = tid; i < RW * Y_DIM; i += RT_THREADS) s.gy[i] = (T)0;
        __syncthreads();
        row_t(s, tid);
        __syncthreads();
        const T* wrow = p.W + row * (long long)W_NUMEL;
        T* dwrow = p.dW + row * (long long)W_NUMEL;
        int step = 0;           // eight input channels (one v) of a path; step i belongs to warp i mod RW
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            constexpr int a = I_IN1[P], b = I_IN2[P], o = I_OUT[P];
            constexpr int D3 = OUT_D[o], MU = IN1_MUL[a], MV = IN2_MUL[b], MW = OUT_MUL[o];
            constexpr int GROUPS = (MU + UG - 1) / UG, STEPS = GROUPS * MV;
            for (int q = (warp + RW - step % RW) % RW; q < STEPS; q += RW) {
                const int v = q / GROUPS, u0 = (q % GROUPS) * UG;       // (a group never straddles a chunk of 32)
                const int uc = u0 / 32, vc = v / 32;
                const int ulen = MU - uc * 32 < 32 ? MU - uc * 32 : 32, vlen = MV - vc * 32 < 32 ? MV - vc * 32 : 32;
                const int n = MU - u0 < UG ? MU - u0 : UG;
                const T* t = s.t + t_offset(P) + (u0 * MV + v) * D3;
                T part[D3][UG];
#pragma unroll
                for (int k = 0; k < D3; ++k)
#pragma unroll
                    for (int i = 0; i < UG; ++i) part[k][i] = (T)0;
                for (int wc = 0; wc < (MW + 31) / 32; ++wc) {
                    const int wlen = MW - wc * 32 < 32 ? MW - wc * 32 : 32;
                    const bool live = lane < wlen;
                    const int off = row_block<P>(uc, vc, wc, ulen, vlen) + ((v - vc * 32) * ulen + u0 - uc * 32) * wlen + lane;
                    T wv[UG], dz[D3];
#pragma unroll
                    for (int i = 0; i < UG; ++i) wv[i] = live && i < n ? __ldcs(wrow + off + i * wlen) : (T)0;
#pragma unroll
                    for (int k = 0; k < D3; ++k) dz[k] = live ? s.zs[OUT_OFF[o] + (wc * 32 + lane) * D3 + k] : (T)0;
#pragma unroll
                    for (int i = 0; i < UG; ++i) {
                        T dw = (T)0;
#pragma unroll
                        for (int k = 0; k < D3; ++k) {
                            part[k][i] = fma(wv[i], dz[k], part[k][i]);
                            if (i < n) dw = fma(t[i * MV * D3 + k], dz[k], dw);
                        }
                        if (live && i < n) __stcs(dwrow + off + i * wlen, dw);
                    }
                }
#pragma unroll
                for (int k = 0; k < D3; ++k) {
                    warp_reduce_8(part[k], lane);
                    if ((lane & 3) == 0 && (lane >> 2) < n) s.dt[t_offset(P) + ((u0 + (lane >> 2)) * MV + v) * D3 + k] = part[k][0];
                }
            }
            step += STEPS;
        });
        __syncthreads();
        // dX[u,i] = sum_{paths, v, j, k} C y[v,j] dT[u,v,k]: one thread per (input irrep, u)
        sfor<0, N_IN1>([&](auto a_) {
            constexpr int a = a_;
            constexpr int D1 = IN1_D[a];
            for (int u = (tid + 32 * a) % RT_THREADS; u < IN1_MUL[a]; u += RT_THREADS) {
                T dx[D1];
#pragma unroll
                for (int i = 0; i < D1; ++i) dx[i] = (T)0;
                sfor<0, N_INSTR>([&](auto p_) {
                    constexpr int P = p_;
                    if constexpr (I_IN1[P] == a) {
                        constexpr int b = I_IN2[P], D3 = OUT_D[I_OUT[P]], MV = IN2_MUL[b];
#pragma unroll 1
                        for (int v = 0; v < MV; ++v) {
                            const T* g = s.dt + t_offset(P) + (u * MV + v) * D3;
                            const T* y = s.ys + IN2_OFF[b] + v * IN2_D[b];
                            sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                                constexpr int N = n_;
                                dx[CG_I[N]] = fma((T)CG_V[N] * g[CG_K[N]], y[CG_J[N]], dx[CG_I[N]]);
                            });
                        }
                    }
                });
#pragma unroll
                for (int i = 0; i < D1; ++i) p.dX[row * X_DIM + IN1_OFF[a] + u * D1 + i] = dx[i];
            }
        });
        // dY[v,j] = sum_{paths, u, i, k} C x[u,i] dT[u,v,k]: a warp per (path, v), lanes along u, one slot per warp
        int pv = 0;
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            constexpr int a = I_IN1[P], b = I_IN2[P], o = I_OUT[P];
            constexpr int D1 = IN1_D[a], D2 = IN2_D[b], D3 = OUT_D[o], MU = IN1_MUL[a], MV = IN2_MUL[b];
            for (int v = 0; v < MV; ++v, ++pv) {
                if ((RW - 1 - pv % RW) != warp) continue;       // (from the last warp down: the first ones do dX)
                T dy[D2];
#pragma unroll
                for (int j = 0; j < D2; ++j) dy[j] = (T)0;
                for (int u = lane; u < MU; u += 32) {
                    const T* x = s.xs + IN1_OFF[a] + u * D1;
                    const T* g = s.dt + t_offset(P) + (u * MV + v) * D3;
                    sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                        constexpr int N = n_;
                        dy[CG_J[N]] = fma((T)CG_V[N] * g[CG_K[N]], x[CG_I[N]], dy[CG_J[N]]);
                    });
                }
#pragma unroll
                for (int j = 0; j < D2; ++j) {
                    const T sum = warp_sum(dy[j]);
                    if (lane == 0) s.gy[warp * Y_DIM + IN2_OFF[b] + v * D2 + j] += sum;
                }
            }
        });
        __syncthreads();
        for (int j = tid; j < Y_DIM; j += RT_THREADS) {
            T sum = (T)0;
            for (int w = 0; w < RW; ++w) sum += s.gy[w * Y_DIM + j];
            p.dY[row * Y_DIM + j] = sum;
        }
        __syncthreads();
    }
}

}  // namespace oeq

#if OEQ_KERNEL == OEQ_K_UVW_ROW_FWD || OEQ_KERNEL == OEQ_K_UVW_ROW_BWD
extern "C" __global__ void __launch_bounds__(oeq::RT_THREADS) oeq_uvw_row_kernel(const oeq::UvwParams p) {
#if OEQ_KERNEL == OEQ_K_UVW_ROW_FWD
    oeq::uvw_row_forward(p);
#else
    oeq::uvw_row_backward(p);
#endif
}
#endif
