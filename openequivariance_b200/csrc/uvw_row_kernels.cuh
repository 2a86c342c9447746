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
// Rows of whole 16-byte pieces take the staged kernels at the end of this file.
#pragma once
#include "uvw_kernels.cuh"

#define OEQ_K_UVW_ROW_FWD 12
#define OEQ_K_UVW_ROW_BWD 13
#define OEQ_K_UVW_STAGED_FWD 14
#define OEQ_K_UVW_STAGED_BWD 15

namespace oeq {

constexpr int RW = ROW_WARPS, RT_THREADS = 32 * ROW_WARPS;
__host__ __device__ constexpr int t_offset(int p) {
    int n = 0;
    for (int q = 0; q < p; ++q) n += IN1_MUL[I_IN1[q]] * IN2_MUL[I_IN2[q]] * OUT_D[I_OUT[q]];
    return n;
}
constexpr int T_ALL = t_offset(N_INSTR);
__host__ __device__ constexpr int t_tasks(int p) {
    int n = 0;
    for (int q = 0; q < p; ++q) n += (IN1_MUL[I_IN1[q]] * IN2_MUL[I_IN2[q]] + 31) / 32;
    return n;
}
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

// T of the row, [path][u][v][k].  A warp has every RW-th task of 32 (u, v) of a path.
__device__ __forceinline__ void row_t(const T* xs, const T* ys, T* t_all, int tid) {
    sfor<0, N_INSTR>([&](auto p_) {
        constexpr int P = p_;
        constexpr int a = I_IN1[P], b = I_IN2[P], o = I_OUT[P];
        constexpr int D1 = IN1_D[a], D2 = IN2_D[b], D3 = OUT_D[o], MV = IN2_MUL[b];
        constexpr int TASKS = (IN1_MUL[a] * MV + 31) / 32, FIRST = t_tasks(P) % RW;
        for (int task = ((tid >> 5) + RW - FIRST) % RW; task < TASKS; task += RW) {
            const int uv = task * 32 + (tid & 31);
            if (IN1_MUL[a] * MV % 32 && uv >= IN1_MUL[a] * MV) continue;
            const int u = uv / MV, v = uv % MV;
            T x[D1], y[D2], t[D3];
#pragma unroll
            for (int i = 0; i < D1; ++i) x[i] = xs[IN1_OFF[a] + u * D1 + i];
#pragma unroll
            for (int j = 0; j < D2; ++j) y[j] = ys[IN2_OFF[b] + v * D2 + j];
#pragma unroll
            for (int k = 0; k < D3; ++k) t[k] = (T)0;
            uvw_cg_forward<P>(x, y, t);
#pragma unroll
            for (int k = 0; k < D3; ++k) t_all[t_offset(P) + uv * D3 + k] = t[k];
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
        row_t(s.xs, s.ys, s.t, tid);
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

// dX of the row, and dY per warp, from dT.
__device__ __forceinline__ void row_dx_dy(const T* xs, const T* ys, const T* dt, T* gy, T* dx_row, int tid, int warp, int lane) {
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
                        const T* g = dt + t_offset(P) + (u * MV + v) * D3;
                        const T* y = ys + IN2_OFF[b] + v * IN2_D[b];
                        sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                            constexpr int N = n_;
                            dx[CG_I[N]] = fma((T)CG_V[N] * g[CG_K[N]], y[CG_J[N]], dx[CG_I[N]]);
                        });
                    }
                }
            });
#pragma unroll
            for (int i = 0; i < D1; ++i) dx_row[IN1_OFF[a] + u * D1 + i] = dx[i];
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
                const T* x = xs + IN1_OFF[a] + u * D1;
                const T* g = dt + t_offset(P) + (u * MV + v) * D3;
                sfor<CG_BEGIN[P], CG_BEGIN[P + 1]>([&](auto n_) {
                    constexpr int N = n_;
                    dy[CG_J[N]] = fma((T)CG_V[N] * g[CG_K[N]], x[CG_I[N]], dy[CG_J[N]]);
                });
            }
#pragma unroll
            for (int j = 0; j < D2; ++j) {
                const T sum = warp_sum(dy[j]);
                if (lane == 0) gy[warp * Y_DIM + IN2_OFF[b] + v * D2 + j] += sum;
            }
        }
    });
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
        row_t(s.xs, s.ys, s.t, tid);
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
        row_dx_dy(s.xs, s.ys, s.dt, s.gy, p.dX + row * X_DIM, tid, warp, lane);
        __syncthreads();
        for (int j = tid; j < Y_DIM; j += RT_THREADS) {
            T sum = (T)0;
            for (int w = 0; w < RW; ++w) sum += s.gy[w * Y_DIM + j];
            p.dY[row * Y_DIM + j] = sum;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- staged rows
//
// The kernels above load a weight where it is used: eight loads in flight per lane, none across the barriers of a row's
// phases, and a path of ten output channels keeps ten lanes of 32 busy.  Here a row's arrays arrive as bulk copies, the
// weights of the next row while this one is at work, three CTAs per SM (about 160 KB of each SM in flight); the work of a
// row is cut into units (path, 32 input channels, 32 output channels) that are dealt to the warps by their length, and a
// warp takes as many input channels side by side as fit beside the output channels.  The weight gradient replaces the
// weights in shared memory and leaves as one copy.
// Rows of X, Y, W and Z of whole 16-byte pieces of which two CTAs fit an SM (uvw_staged_smem in the runtime); arrays that do not
// start on a 16-byte boundary are copied by all threads when the row's turn comes.
// 2 011 rows of 10x1o+10x1e+48x0e+48x0o with 1x0e+1x1o, FP32, both launches 64 -> 43 us (weights and their gradients take 26 at the
// copy rate).  Backward: issue 52 %, then barriers and the answers of shared memory.
#if OEQ_KERNEL == OEQ_K_UVW_STAGED_FWD || OEQ_KERNEL == OEQ_K_UVW_STAGED_BWD
constexpr bool STAGED_BWD = OEQ_KERNEL == OEQ_K_UVW_STAGED_BWD;
constexpr int ROW_STAGE = W_NUMEL + X_DIM + Y_DIM + (STAGED_BWD ? Z_DIM : 0);      // values: W, X, Y, dZ
constexpr int ERR_ROW_FULL = 41;

__host__ __device__ constexpr int in_chunks(int p) { return (IN1_MUL[I_IN1[p]] + 31) / 32; }
__host__ __device__ constexpr int out_chunks(int p) { return (OUT_MUL[I_OUT[p]] + 31) / 32; }
__host__ __device__ constexpr int chunk_len(int mul, int c) { return mul - 32 * c < 32 ? mul - 32 * c : 32; }
// Forward units: (path, chunk of input channels, chunk of output channels).  Backward: (path, 16 input channels, v): a warp
// reads the places of its units from a table, and one body serves all units of the same widths.  With a body per unit the
// backward kernel waited for instructions longer than for everything else (8 of 15 stalled warps per issue, 42 us where it takes
// 32 now, under ncu); the forward kernel's bodies are short (15 us, through a table 27).
constexpr int BU = 16;
__host__ __device__ constexpr int bwd_groups(int p) { return (IN1_MUL[I_IN1[p]] + BU - 1) / BU; }
__host__ __device__ constexpr int path_units(int p) { return STAGED_BWD ? bwd_groups(p) * IN2_MUL[I_IN2[p]] : in_chunks(p) * out_chunks(p); }
__host__ __device__ constexpr int units_before(int p_end) {
    int n = 0;
    for (int p = 0; p < p_end; ++p) n += path_units(p);
    return n;
}
constexpr int N_UNITS = units_before(N_INSTR);
// Input channels that a warp takes side by side beside n output channels (backward: segments of a power of two, for the
// sums over the lanes).
__host__ __device__ constexpr int seg_len(int n) { return n <= 8 ? 8 : (n <= 16 ? 16 : 32); }
__host__ __device__ constexpr int side_by_side(int n) { return STAGED_BWD ? 32 / seg_len(n) : 32 / n; }
struct Unit {
    int w, t, u0, v, out, body;         // places of the weights, T, first channel of its chunk of 32, v, dZ; unit with its body
    int d3, mv, mw, us, ulen;           // (constants of a body:) components, multiplicities, channels of the unit, of its chunk
    int cost;
};
struct UnitTable {
    Unit unit[N_UNITS], dealt[N_UNITS];     // in order, and by warp
    int owner[N_UNITS], begin[RW + 1];      // warp of a unit, first unit of a warp
};
constexpr UnitTable deal_units() {
    Unit all[N_UNITS] = {};
    int n = 0;
    for (int p = 0; p < N_INSTR; ++p) {
        const int o = I_OUT[p], d3 = OUT_D[o], mu = IN1_MUL[I_IN1[p]], mv = IN2_MUL[I_IN2[p]], mw = OUT_MUL[o];
        for (int i = 0; i < path_units(p); ++i, ++n) {
            Unit& x = all[n];
            x.d3 = d3; x.mv = mv; x.mw = mw;
            if (STAGED_BWD) {
                const int u0 = i / mv * BU;
                x.us = mu - u0 < BU ? mu - u0 : BU;
                x.ulen = chunk_len(mu, u0 / 32);
                x.u0 = u0 & 31;
                x.v = i % mv;
                x.w = W_OFF[p] + u0 / 32 * 32 * mv * mw;
                x.t = t_offset(p) + (u0 * mv + x.v) * d3;
                x.out = OUT_OFF[o];
                for (int wc = 0; wc < out_chunks(p); ++wc) {
                    const int ul = side_by_side(chunk_len(mw, wc));
                    x.cost += (x.us + 8 * ul - 1) / (8 * ul) * (16 + 66 * d3);
                }
                x.body = n;
                for (int m = n - 1; m >= 0; --m)
                    if (all[m].d3 == d3 && all[m].mv == mv && all[m].mw == mw && all[m].us == x.us && all[m].ulen == x.ulen) x.body = m;
            } else {
                const int ul = side_by_side(chunk_len(mw, i % out_chunks(p)));
                x.cost = 8 + (chunk_len(mu, i / out_chunks(p)) + ul - 1) / ul * (2 + 2 * d3) * mv;
                x.body = n;
            }
        }
    }
    // longest first, each to the warp with the least to do
    UnitTable t{};
    int load[RW] = {};
    bool taken[N_UNITS] = {};
    for (int k = 0; k < N_UNITS; ++k) {
        int best = -1, w = 0;
        for (int i = 0; i < N_UNITS; ++i)
            if (!taken[i] && (best < 0 || all[i].cost > all[best].cost)) best = i;
        for (int i = 1; i < RW; ++i)
            if (load[i] < load[w]) w = i;
        taken[best] = true;
        t.unit[k] = all[k];
        t.owner[best] = w;
        load[w] += all[best].cost;
    }
    int k = 0;
    for (int w = 0; w < RW; ++w) {
        t.begin[w] = k;
        for (int i = 0; i < N_UNITS; ++i)
            if (t.owner[i] == w) t.dealt[k++] = all[i];
    }
    t.begin[RW] = k;
    return t;
}
constexpr UnitTable UNITS = deal_units();
// Forward: sums of a path's chunks, [input channel side by side][output channel][component].
__host__ __device__ constexpr int part_offset(int unit_end) {
    int n = 0;
    for (int p = 0; p < N_INSTR; ++p)
        for (int uc = 0; uc < in_chunks(p); ++uc)
            for (int wc = 0; wc < out_chunks(p); ++wc) {
                if (units_before(p) + uc * out_chunks(p) + wc >= unit_end) return n;
                const int wlen = chunk_len(OUT_MUL[I_OUT[p]], wc);
                n += 32 / wlen * wlen * OUT_D[I_OUT[p]];
            }
    return n;
}
struct StagedSmem {
    T *first, *t, *extra;        // extra: sums of the units (forward), dT and dY per warp of two rows (backward)
    Unit* units;                    // backward
    unsigned long long* full;
    __device__ explicit StagedSmem(unsigned char* raw) {
        first = reinterpret_cast<T*>(raw);
        t = first + 2 * ROW_STAGE;
        extra = t + r4(T_ALL);
        units = reinterpret_cast<Unit*>(extra + r4(STAGED_BWD ? r4(T_ALL) + 2 * RW * Y_DIM : part_offset(N_UNITS)));
        full = reinterpret_cast<unsigned long long*>(units + (STAGED_BWD ? N_UNITS : 0));
    }
    __device__ __forceinline__ T* stage(int b) const { return first + b * ROW_STAGE; }
};

// (one thread) a row's arrays into a stage
__device__ __forceinline__ void stage_row(const UvwParams& p, const StagedSmem& s, int b, long long row, unsigned long long stream) {
    T* st = s.stage(b);
    mbar_arrive_expect_tx(s.full + b, ROW_STAGE * (unsigned)sizeof(T));
    bulk_g2s_hint(st, p.W + row * W_NUMEL, W_NUMEL * sizeof(T), s.full + b, stream);
    bulk_g2s(st + W_NUMEL, p.X + row * X_DIM, X_DIM * sizeof(T), s.full + b);
    bulk_g2s(st + W_NUMEL + X_DIM, p.Y + row * Y_DIM, Y_DIM * sizeof(T), s.full + b);
    if constexpr (STAGED_BWD) bulk_g2s(st + W_NUMEL + X_DIM + Y_DIM, p.dZ + row * Z_DIM, Z_DIM * sizeof(T), s.full + b);
}

// (all threads) the same without bulk copies; the caller lets the threads meet
__device__ __forceinline__ void copy_row(const UvwParams& p, T* st, long long row, int tid) {
    for (int i = tid; i < W_NUMEL; i += RT_THREADS) st[i] = __ldcs(p.W + row * W_NUMEL + i);
    for (int i = tid; i < X_DIM; i += RT_THREADS) st[W_NUMEL + i] = p.X[row * X_DIM + i];
    for (int i = tid; i < Y_DIM; i += RT_THREADS) st[W_NUMEL + X_DIM + i] = p.Y[row * Y_DIM + i];
    if constexpr (STAGED_BWD)
        for (int i = tid; i < Z_DIM; i += RT_THREADS) st[W_NUMEL + X_DIM + Y_DIM + i] = p.dZ[row * Z_DIM + i];
}

#if OEQ_KERNEL == OEQ_K_UVW_STAGED_FWD
template <int P, int UC, int WC>
__device__ __forceinline__ void staged_forward_unit(const T* wt, const T* t_all, T* part, int lane) {
    constexpr int D3 = OUT_D[I_OUT[P]], MU = IN1_MUL[I_IN1[P]], MV = IN2_MUL[I_IN2[P]], MW = OUT_MUL[I_OUT[P]];
    constexpr int ULEN = chunk_len(MU, UC), WLEN = chunk_len(MW, WC), UL = 32 / WLEN;
    const int du = lane / WLEN;
    T acc[D3];
#pragma unroll
    for (int k = 0; k < D3; ++k) acc[k] = (T)0;
#pragma unroll 1
    for (int vc = 0; vc < (MV + 31) / 32; ++vc) {
        const int vlen = chunk_len(MV, vc);
        const T* w = wt + row_block<P>(UC, vc, WC, ULEN, vlen);
#pragma unroll 1
        for (int vl = 0; vl < vlen; ++vl, w += ULEN * WLEN) {
            const T* t = t_all + t_offset(P) + ((UC * 32 + du) * MV + vc * 32 + vl) * D3;
#pragma unroll
            for (int u0 = 0; u0 < ULEN; u0 += UL) {
                if (lane < UL * WLEN && (u0 + UL <= ULEN || u0 + du < ULEN)) {
                    const T q = w[u0 * WLEN + lane];
#pragma unroll
                    for (int k = 0; k < D3; ++k) acc[k] = fma(q, t[u0 * MV * D3 + k], acc[k]);
                }
            }
        }
    }
    if (lane < UL * WLEN) {
#pragma unroll
        for (int k = 0; k < D3; ++k) part[lane * D3 + k] = acc[k];
    }
}

__device__ void uvw_staged_forward(const UvwParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StagedSmem s(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long stream = l2_policy_evict_first();
    if (tid == 0) {
        mbar_init(s.full, 1);
        mbar_init(s.full + 1, 1);
        fence_mbar_init();
        for (int b = 0; b < 2 && p.bulk; ++b)
            if (blockIdx.x + b * (long long)gridDim.x < p.batch) stage_row(p, s, b, blockIdx.x + b * (long long)gridDim.x, stream);
    }
    __syncthreads();
    int it = 0;
    for (long long row = blockIdx.x; row < p.batch; row += gridDim.x, ++it) {
        const int b = it & 1;
        T* st = s.stage(b);
        bool ok = true;
        if (p.bulk) {
            ok = mbar_wait(s.full + b, (unsigned)(it >> 1) & 1, p.status, ERR_ROW_FULL);
        } else {
            copy_row(p, st, row, tid);
            __syncthreads();
        }
        if (ok) row_t(st + W_NUMEL, st + W_NUMEL + X_DIM, s.t, tid);
        if (!__syncthreads_and(ok)) {
            // (the copies in flight must land before the CTA's shared memory goes to another one)
            if (tid == 0 && p.bulk && row + gridDim.x < p.batch) mbar_wait(s.full + (b ^ 1), (unsigned)((it + 1) >> 1) & 1, p.status, ERR_ROW_FULL);
            return;
        }
        sfor<0, N_INSTR>([&](auto p_) {
            constexpr int P = p_;
            sfor<0, in_chunks(P) * out_chunks(P)>([&](auto c_) {
                constexpr int UC = c_ / out_chunks(P), WC = c_ % out_chunks(P), UNIT = units_before(P) + c_;
                constexpr int OWNER = UNITS.owner[UNIT];
                if (warp == OWNER) staged_forward_unit<P, UC, WC>(st, s.t, s.extra + part_offset(UNIT), lane);
            });
        });
        __syncthreads();        // sums complete; the stage has been read
        if (tid == 0 && p.bulk && row + 2ll * gridDim.x < p.batch) stage_row(p, s, b, row + 2ll * gridDim.x, stream);
        T* zrow = p.Z + row * (long long)Z_DIM;
        sfor<0, N_OUT>([&](auto o_) {
            constexpr int o = o_;
            constexpr int D3 = OUT_D[o], MW = OUT_MUL[o];
            for (int e = (tid + 64 * o) % RT_THREADS; e < MW * D3; e += RT_THREADS) {
                T sum = (T)0;
                sfor<0, N_INSTR>([&](auto p_) {
                    constexpr int P = p_;
                    if constexpr (I_OUT[P] == o) {
                        sfor<0, in_chunks(P) * out_chunks(P)>([&](auto c_) {
                            constexpr int WC = c_ % out_chunks(P), OFF = part_offset(units_before(P) + c_);
                            constexpr int WLEN = chunk_len(MW, WC), UL = 32 / WLEN;
                            if (out_chunks(P) == 1 || e / (32 * D3) == WC) {
#pragma unroll
                                for (int d = 0; d < UL; ++d) sum += s.extra[OFF + d * WLEN * D3 + e - 32 * WC * D3];
                            }
                        });
                    }
                });
                zrow[OUT_OFF[o] + e] = sum;
            }
        });
    }
}

#else
__device__ const UnitTable UNITS_DEV = deal_units();

// Sum v[0..8) over segments of SEG lanes in a fixed order; within a segment lane l ends with the total of value
// l / (SEG / 8) in v[0].
template <int SEG, class VA>
__device__ __forceinline__ void segment_reduce_8(VA& v, int lane) {
#pragma unroll
    for (int off = SEG / 2, half = 4; off > 0; off >>= 1, half >>= 1) {
        if (half > 0) {
            const bool upper = (lane & off) != 0;
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m < half) {
                    const T send = upper ? v[m] : v[m + half], keep = upper ? v[m + half] : v[m];
                    v[m] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        }
    }
}

// Some input channels of a path with component v of the second input: dW in the place of W, and dT.  BODY: a unit of the same
// widths.
template <int BODY>
__device__ __forceinline__ void staged_backward_unit(const Unit& x, T* wt, const T* dz_row, const T* t_all, T* dt_all, int lane) {
    constexpr int D3 = UNITS.unit[BODY].d3, MV = UNITS.unit[BODY].mv, MW = UNITS.unit[BODY].mw, US = UNITS.unit[BODY].us, ULEN = UNITS.unit[BODY].ulen;
    const T* t = t_all + x.t;
    T* dt = dt_all + x.t;
    const int vc = MV > 1 ? x.v >> 5 : 0, vl = MV > 1 ? x.v & 31 : 0, vlen = MV > 32 ? chunk_len(MV, vc) : MV;
    sfor<0, (MW + 31) / 32>([&](auto wc_) {
        constexpr int WC = wc_, WLEN = chunk_len(MW, WC), SEG = seg_len(WLEN), UL = 32 / SEG;
        const int du = lane / SEG, wl = lane % SEG;
        const bool live = wl < WLEN;
        T* w = wt + x.w + ULEN * (vc * 32 * MW + vlen * 32 * WC) + (vl * ULEN + x.u0 + du) * WLEN + wl;
        T dz[D3];
#pragma unroll
        for (int k = 0; k < D3; ++k) dz[k] = live ? dz_row[x.out + (WC * 32 + wl) * D3 + k] : (T)0;
#pragma unroll
        for (int u1 = 0; u1 < US; u1 += 8 * UL) {       // value i of a lane: input channel u1 + du + UL i of the unit
            T part[D3][8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int u = u1 + UL * i;
                const bool on = live && (u + UL <= US || u + du < US);
                const T q = u < US && on ? w[u * WLEN] : (T)0;
                T dw = (T)0;
#pragma unroll
                for (int k = 0; k < D3; ++k) {
                    part[k][i] = q * dz[k];
                    if (u < US && on) dw = fma(t[(u + du) * MV * D3 + k], dz[k], dw);
                }
                if (u < US && on) w[u * WLEN] = dw;
            }
#pragma unroll
            for (int k = 0; k < D3; ++k) {
                segment_reduce_8<SEG>(part[k], lane);
                const int u = u1 + du + UL * (wl / (SEG / 8));
                if (wl % (SEG / 8) == 0 && u < US) {
                    T* d = dt + u * MV * D3 + k;
                    *d = WC ? *d + part[k][0] : part[k][0];
                }
            }
        }
        if (WC + 1 < (MW + 31) / 32) __syncwarp();      // (another lane may add the next chunk's sums)
    });
}

__device__ void uvw_staged_backward(const UvwParams& p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const StagedSmem s(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long stream = l2_policy_evict_first();
    T* const dt = s.extra;
    for (int i = tid; i < N_UNITS * (int)(sizeof(Unit) / 4); i += RT_THREADS)
        reinterpret_cast<int*>(s.units)[i] = reinterpret_cast<const int*>(UNITS_DEV.dealt)[i];
    const int mine = UNITS_DEV.begin[warp], end = UNITS_DEV.begin[warp + 1];
    if (tid == 0) {
        mbar_init(s.full, 1);
        mbar_init(s.full + 1, 1);
        fence_mbar_init();
        if (p.bulk && blockIdx.x < p.batch) stage_row(p, s, 0, blockIdx.x, stream);
    }
    __syncthreads();
    int it = 0;
    for (long long row = blockIdx.x; row < p.batch; row += gridDim.x, ++it) {
        const int b = it & 1;
        T* st = s.stage(b);
        T* gy = s.extra + r4(T_ALL) + b * RW * Y_DIM;
        bool ok = true;
        if (p.bulk) {
            ok = mbar_wait(s.full + b, (unsigned)(it >> 1) & 1, p.status, ERR_ROW_FULL);
        } else {
            copy_row(p, st, row, tid);
            __syncthreads();
        }
        for (int i = tid; i < RW * Y_DIM; i += RT_THREADS) gy[i] = (T)0;
        if (ok) row_t(st + W_NUMEL, st + W_NUMEL + X_DIM, s.t, tid);
        if (!__syncthreads_and(ok)) break;
        if (tid == 0 && p.bulk && row + gridDim.x < p.batch) {
            bulk_wait_read<0>();        // the weight gradient of the row before has left the other stage
            stage_row(p, s, b ^ 1, row + gridDim.x, stream);
        }
#pragma unroll 1
        for (int n = mine; n < end; ++n) {
            const Unit& x = s.units[n];
            sfor<0, N_UNITS>([&](auto b_) {
                if constexpr (UNITS.unit[b_].body == b_) {
                    if (x.body == b_) staged_backward_unit<b_>(x, st, st + W_NUMEL + X_DIM + Y_DIM, s.t, dt, lane);
                }
            });
        }
        fence_async_smem();
        __syncthreads();
        if (!p.bulk) {
            for (int i = tid; i < W_NUMEL; i += RT_THREADS) __stcs(p.dW + row * W_NUMEL + i, st[i]);
        } else if (tid == 0) {
            bulk_s2g(p.dW + row * W_NUMEL, st, W_NUMEL * sizeof(T));
            bulk_commit();
        }
        row_dx_dy(st + W_NUMEL, st + W_NUMEL + X_DIM, dt, gy, p.dX + row * X_DIM, tid, warp, lane);
        __syncthreads();
        for (int j = tid; j < Y_DIM; j += RT_THREADS) {
            T sum = (T)0;
            for (int w = 0; w < RW; ++w) sum += gy[w * Y_DIM + j];
            p.dY[row * Y_DIM + j] = sum;
        }
    }
    if (tid == 0) bulk_wait_all<0>();
}
#endif
#endif

}  // namespace oeq

#if OEQ_KERNEL == OEQ_K_UVW_STAGED_FWD
extern "C" __global__ void __launch_bounds__(oeq::RT_THREADS) oeq_uvw_row_kernel(const oeq::UvwParams p) { oeq::uvw_staged_forward(p); }
#elif OEQ_KERNEL == OEQ_K_UVW_STAGED_BWD
extern "C" __global__ void __launch_bounds__(oeq::RT_THREADS) oeq_uvw_row_kernel(const oeq::UvwParams p) { oeq::uvw_staged_backward(p); }
#elif OEQ_KERNEL == OEQ_K_UVW_ROW_FWD || OEQ_KERNEL == OEQ_K_UVW_ROW_BWD
extern "C" __global__ void __launch_bounds__(oeq::RT_THREADS) oeq_uvw_row_kernel(const oeq::UvwParams p) {
#if OEQ_KERNEL == OEQ_K_UVW_ROW_FWD
    oeq::uvw_row_forward(p);
#else
    oeq::uvw_row_backward(p);
#endif
}
#endif
