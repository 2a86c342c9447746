// Host runtime behind the C ABI (include/oeq_b200.h).
//
// Replaces the reference's native layer (openequivariance/extension/:
// JITTPImpl / JITConvImpl in tensorproducts.hpp:50-98 and convolution.hpp:94-176,
// the NVRTC + driver wrapper CUJITKernel in util/backend_cuda.hpp:139-300) and the
// launch-shape half of its scheduler (implementations/ComputationSchedule.py:232-425).
//
// For a problem it (1) picks the thread mapping (channels per group, path
// partitions, groups per CTA), (2) emits a small header of constexpr tables that
// describes the problem -- irreps, instructions, Clebsch-Gordan nonzeros scaled by
// the path weights, the mapping -- (3) compiles the hand-written kernel templates
// in csrc/*.cuh against it with NVRTC for sm_100a, caching the CUBIN on disk, and
// (4) launches through the CUDA runtime's library API on the caller's stream.
// No kernel body is generated; no CPU fallback exists.

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nvrtc.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <mutex>
#include <set>
#include <sstream>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/oeq_b200.h"
#include "oeq_common.cuh"

namespace {

thread_local std::string g_error;
int fail(int code, const std::string& msg) {
    g_error = msg;
    return code;
}
#define OEQ_CUDA(expr)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (expr);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return fail(OEQ_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_));      \
    } while (0)

std::mutex g_mutex;
std::string g_kernel_dir, g_cache_dir;

std::string library_dir() {
    Dl_info info;
    if (dladdr(reinterpret_cast<void*>(&library_dir), &info) && info.dli_fname) {
        std::string p(info.dli_fname);
        size_t slash = p.find_last_of('/');
        return slash == std::string::npos ? std::string(".") : p.substr(0, slash);
    }
    return ".";
}
std::string kernel_dir() {
    if (!g_kernel_dir.empty()) return g_kernel_dir;
    if (const char* e = getenv("OEQ_B200_KERNEL_DIR")) return e;
    return library_dir() + "/csrc";
}
std::string cache_dir() {
    if (!g_cache_dir.empty()) return g_cache_dir;
    if (const char* e = getenv("OEQ_B200_CACHE_DIR")) return e;
    return library_dir() + "/_kcache";
}
int env_int(const char* name, int fallback) {
    const char* e = getenv(name);
    return e && *e ? atoi(e) : fallback;
}

// ------------------------------------------------------------------ NVRTC, loaded on first use

struct Nvrtc {
    void* lib = nullptr;
    decltype(&nvrtcCreateProgram) create = nullptr;
    decltype(&nvrtcCompileProgram) compile = nullptr;
    decltype(&nvrtcGetCUBINSize) cubin_size = nullptr;
    decltype(&nvrtcGetCUBIN) cubin = nullptr;
    decltype(&nvrtcGetProgramLogSize) log_size = nullptr;
    decltype(&nvrtcGetProgramLog) log = nullptr;
    decltype(&nvrtcDestroyProgram) destroy = nullptr;
    decltype(&nvrtcGetErrorString) error_string = nullptr;
};
Nvrtc g_nvrtc;

int load_nvrtc() {
    if (g_nvrtc.lib) return OEQ_OK;
    const char* names[] = {"libnvrtc.so.12", "/usr/local/cuda/lib64/libnvrtc.so.12", "libnvrtc.so",
                           "/usr/local/cuda/lib64/libnvrtc.so"};
    void* lib = nullptr;
    for (const char* n : names) {
        lib = dlopen(n, RTLD_NOW | RTLD_LOCAL);
        if (lib) break;
    }
    if (!lib) return fail(OEQ_ERR_COMPILE, "cannot load libnvrtc (needed to specialise kernels)");
#define OEQ_SYM(field, name)                                                      \
    g_nvrtc.field = reinterpret_cast<decltype(g_nvrtc.field)>(dlsym(lib, name));  \
    if (!g_nvrtc.field) return fail(OEQ_ERR_COMPILE, std::string("libnvrtc lacks ") + name);
    OEQ_SYM(create, "nvrtcCreateProgram")
    OEQ_SYM(compile, "nvrtcCompileProgram")
    OEQ_SYM(cubin_size, "nvrtcGetCUBINSize")
    OEQ_SYM(cubin, "nvrtcGetCUBIN")
    OEQ_SYM(log_size, "nvrtcGetProgramLogSize")
    OEQ_SYM(log, "nvrtcGetProgramLog")
    OEQ_SYM(destroy, "nvrtcDestroyProgram")
    OEQ_SYM(error_string, "nvrtcGetErrorString")
#undef OEQ_SYM
    g_nvrtc.lib = lib;
    return OEQ_OK;
}

// ------------------------------------------------------------------ problem model

struct Irrep {
    int mul, l, parity, dim, off;
};
struct Instr {
    int i1, i2, io, mode;
    double pw;
    std::vector<int> ci, cj, ck;
    std::vector<double> cv;
    int w_off;  // first weight of the instruction (same in e3nn and kernel order)
    long long cost() const { return (long long)cv.size(); }
};
struct Problem {
    std::vector<Irrep> in1, in2, out;
    std::vector<Instr> instr;
    int dtype = 0, shared = 0, mode = 0;
    bool unit_y = false;        // the second input is the number 1 for every row (no array)
    bool transposed_w = false;  // the weight array is that of the problem with first input and output exchanged, and an
                                // output block joins several of its paths (subs, per instruction)
    struct Sub { int start, mul, w_off; };
    std::vector<std::vector<Sub>> subs;
    int unit = 0;               // no weight array: every weight is 1 (shared_weights == 2 in the descriptor)
    int x_dim = 0, y_dim = 0, z_dim = 0, w_numel = 0;
    int elem() const { return dtype == OEQ_F64 ? 8 : 4; }
};

int ingest_irreps(const oeq_irrep* src, int n, std::vector<Irrep>& dst, int& dim, const char* what) {
    if (n < 0 || (n > 0 && !src)) return fail(OEQ_ERR_INVALID, std::string(what) + ": null irreps");
    int off = 0;
    for (int i = 0; i < n; ++i) {
        if (src[i].mul < 0 || src[i].l < 0 || (src[i].parity != 1 && src[i].parity != -1))
            return fail(OEQ_ERR_INVALID, std::string(what) + ": bad irrep entry");
        Irrep r{src[i].mul, src[i].l, src[i].parity, 2 * src[i].l + 1, off};
        off += r.mul * r.dim;
        dst.push_back(r);
    }
    dim = off;
    return OEQ_OK;
}

int ingest(const oeq_problem_desc* d, Problem& p) {
    if (!d) return fail(OEQ_ERR_INVALID, "null problem descriptor");
    if (d->dtype != OEQ_F32 && d->dtype != OEQ_F64) return fail(OEQ_ERR_INVALID, "dtype must be OEQ_F32 or OEQ_F64");
    p.dtype = d->dtype;
    p.unit = d->shared_weights == 2 ? 1 : 0;
    p.shared = (d->shared_weights && !p.unit) ? 1 : 0;
    int rc;
    if ((rc = ingest_irreps(d->in1, d->n_in1, p.in1, p.x_dim, "irreps_in1"))) return rc;
    if ((rc = ingest_irreps(d->in2, d->n_in2, p.in2, p.y_dim, "irreps_in2"))) return rc;
    if ((rc = ingest_irreps(d->out, d->n_out, p.out, p.z_dim, "irreps_out"))) return rc;
    if (d->n_instr <= 0 || !d->instr)
        return fail(OEQ_ERR_INVALID, "Tensor product problem has no valid intructions!");
    p.mode = d->instr[0].mode;
    if (p.mode != OEQ_MODE_UVU && p.mode != OEQ_MODE_UVW)
        return fail(OEQ_ERR_UNSUPPORTED, "connection mode must be 'uvu' or 'uvw'");
    int w = 0;
    for (int n = 0; n < d->n_instr; ++n) {
        const oeq_instruction& s = d->instr[n];
        if (s.mode != p.mode) return fail(OEQ_ERR_UNSUPPORTED, "all instructions must share one connection mode");
        if (s.i_in1 < 0 || s.i_in1 >= d->n_in1 || s.i_in2 < 0 || s.i_in2 >= d->n_in2 || s.i_out < 0 ||
            s.i_out >= d->n_out)
            return fail(OEQ_ERR_INVALID, "instruction index out of range");
        const Irrep &a = p.in1[s.i_in1], &b = p.in2[s.i_in2], &c = p.out[s.i_out];
        if (a.parity * b.parity != c.parity || c.l < std::abs(a.l - b.l) || c.l > a.l + b.l)
            return fail(OEQ_ERR_INVALID, "instruction violates the selection rules");
        if (p.mode == OEQ_MODE_UVU && a.mul != c.mul)
            return fail(OEQ_ERR_INVALID, "'uvu' needs equal multiplicities of the first input and the output");
        Instr t;
        t.i1 = s.i_in1; t.i2 = s.i_in2; t.io = s.i_out; t.mode = s.mode; t.pw = s.path_weight;
        if (s.cg_nnz < 0 || (s.cg_nnz > 0 && (!s.cg_i || !s.cg_j || !s.cg_k || !s.cg_value)))
            return fail(OEQ_ERR_INVALID, "instruction has a malformed Clebsch-Gordan list");
        for (int z = 0; z < s.cg_nnz; ++z) {
            if (s.cg_i[z] < 0 || s.cg_i[z] >= a.dim || s.cg_j[z] < 0 || s.cg_j[z] >= b.dim || s.cg_k[z] < 0 ||
                s.cg_k[z] >= c.dim)
                return fail(OEQ_ERR_INVALID, "Clebsch-Gordan index out of range");
            t.ci.push_back(s.cg_i[z]); t.cj.push_back(s.cg_j[z]); t.ck.push_back(s.cg_k[z]);
            t.cv.push_back(s.cg_value[z] * s.path_weight);
        }
        t.w_off = w;
        w += a.mul * b.mul * (p.mode == OEQ_MODE_UVW ? c.mul : 1);
        p.instr.push_back(std::move(t));
    }
    p.w_numel = w;
    return OEQ_OK;
}

// ------------------------------------------------------------------ thread mapping for the "uvu" kernels

enum Kind { K_FWD_BATCH = 0, K_BWD_BATCH, K_FWD_DET, K_BWD_DET, K_FWD_ATOMIC, K_BWD_ATOMIC, K_COUNT };
bool kind_is_bwd(int k) { return k & 1; }
bool kind_is_batch(int k) { return k < 2; }

constexpr int SMEM_LIMIT = 232448;  // opt-in dynamic shared memory per CTA on sm_100
int pad16(int b) { return (b + 15) / 16 * 16; }

struct Mapping {
    int mulg = 32, nch = 1, ps = 1, ng = 1, producer = 0, min_ctas = 1;
    int nph = 1;                              // backward staging in phases (see uvu_kernels.cuh)
    bool tc_tables = false;                   // emit the tables of the tensor-core forward pass
    std::vector<int> z_ph_begin, w_ph_begin;  // nph + 1 column / weight boundaries
    std::vector<int> phase_of_instr;
    std::vector<int> part_of_out, part_of_instr, zr_off, xr_off;
    int zpc_max = 1, xpc = 1;
    int stage_bytes = 0, extra_bytes = 0, sw_bytes = 0;
    int helper_warps = 0;                     // receiver-order backward: warps that sum the previous block's rows
    int gz_regs = 1 << 20, gz_smem_values = 0; // receiver-order backward: dZ values in registers / parked in shared memory
    int epi = 1;                              // edges per staged item (uvu_kernels.cuh, EPI)
    int stage_cap = 4;                        // most stages a group takes
    int chunk_floor = 32;                     // smallest chunk of consecutive edges a launch may deal out
    int slice_warps = 0, n_slice = 1;         // slice kernels (uvu_slice_kernels.cuh): warps per CTA (0: not one of them)
    bool slice_full = false;
    bool slice_outer = false;       // no weights: sums of products per receiver
    int slice_cpl = 1;              // channels per lane
    bool slice_one = false;         // one edge at a time, and per stage
    int slice_stages = 2, slice_smem = 0, slice_regs = 0;
    int threads() const { return ng * mulg * ps + 32 * ng * producer + 32 * helper_warps; }
    int fixed_bytes(int stages) const { return ng * stages * (16 + 8 * (epi > 1 ? 4 + 2 * epi : 4)) + ng * 128 + sw_bytes; }
    int smem(int stages) const { return fixed_bytes(stages) + ng * (stages * stage_bytes + extra_bytes); }
    int max_stages() const {
        int s = 0;
        while (s < stage_cap && smem(s + 1) <= SMEM_LIMIT) ++s;
        return s;
    }
};

void assign_partitions(const Problem& p, bool bwd, Mapping& m) {
    // longest-processing-time first; forward units are output irreps, backward units instructions
    const int n_units = bwd ? (int)p.instr.size() : (int)p.out.size();
    std::vector<long long> cost(n_units, 0);
    for (size_t i = 0; i < p.instr.size(); ++i) {
        long long c = p.instr[i].cost() * p.in2[p.instr[i].i2].mul + 2;
        cost[bwd ? (int)i : p.instr[i].io] += c;
    }
    std::vector<int> order(n_units);
    for (int i = 0; i < n_units; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<long long> load(m.ps, 0);
    std::vector<int> part(n_units, 0);
    for (int unit : order) {
        int best = 0;
        for (int q = 1; q < m.ps; ++q)
            if (load[q] < load[best]) best = q;
        part[unit] = best;
        load[best] += cost[unit];
    }
    m.part_of_out.assign(p.out.size(), 0);
    m.part_of_instr.assign(p.instr.size(), 0);
    if (bwd) {
        m.part_of_instr = part;
    } else {
        m.part_of_out = part;
        for (size_t i = 0; i < p.instr.size(); ++i) m.part_of_instr[i] = part[p.instr[i].io];
    }
    // register offsets of the per-channel accumulators
    m.zr_off.assign(p.out.size(), 0);
    std::vector<int> fill(m.ps, 0);
    for (size_t o = 0; o < p.out.size(); ++o) {
        int q = bwd ? 0 : m.part_of_out[o];
        m.zr_off[o] = fill[q];
        fill[q] += p.out[o].dim;
    }
    m.zpc_max = std::max(1, *std::max_element(fill.begin(), fill.end()));
    m.xr_off.assign(p.in1.size(), 0);
    int x = 0;
    for (size_t a = 0; a < p.in1.size(); ++a) {
        m.xr_off[a] = x;
        x += p.in1[a].dim;
    }
    m.xpc = std::max(1, x);
}

// Narrow self-staging groups (one warp per group) of the receiver-order walks stage runs of consecutive edges:
// the per-item fixed cost (list walk, copies, hand-off) is shared by up to `epi` edges.  Re-fits the group count.
void apply_edges_per_item(const Problem& p, Mapping& m, int extra_per_group) {
    m.epi = 1;
    const int want = env_int("OEQ_B200_EPI", 2);
    if (want <= 1 || want > 8 || m.producer || m.mulg * m.ps > 32 || p.shared) return;
    const int e = p.elem();
    const int xb = pad16(p.x_dim * e);
    const int wrow = p.unit ? 0 : p.w_numel * e;
    Mapping t = m;
    t.epi = want;
    t.stage_bytes = want * xb + pad16(want * p.y_dim * e) + pad16(want * wrow);
    t.extra_bytes = extra_per_group;
    // two stages of `want` edges keep as many edges in flight as four stages of one
    t.stage_cap = std::max(2, std::min(4, env_int("OEQ_B200_EPI_STAGES", 2)));
    while (t.ng > 1 && t.smem(t.stage_cap) > SMEM_LIMIT) --t.ng;
    if (t.smem(t.stage_cap) > SMEM_LIMIT) return;
    m = t;
    const int stages = std::min(m.max_stages(), env_int("OEQ_B200_STAGES", 4));
    const int by_smem = stages >= 2 ? SMEM_LIMIT / (m.smem(stages) + 1024) : 1;
    m.min_ctas = std::max(1, std::min({by_smem, 2048 / m.threads(), 2}));
}

int choose_mapping(const Problem& p, int kind, Mapping& m) {
    const bool bwd = kind_is_bwd(kind), batch = kind_is_batch(kind);
    int maxmul = 1;
    for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
    for (const Irrep& r : p.out) maxmul = std::max(maxmul, r.mul);
    m.mulg = std::min((maxmul + 31) / 32 * 32, 256);
    m.nch = (maxmul + m.mulg - 1) / m.mulg;
    const int e = p.elem();
    const int xb = pad16(p.x_dim * e), yb = pad16(p.y_dim * e), zb = pad16(p.z_dim * e);
    const int wb = (p.shared || p.unit) ? 0 : pad16(p.w_numel * e);
    m.sw_bytes = p.shared ? pad16(p.w_numel * e) : 0;
    m.stage_bytes = xb + yb + wb + (bwd ? zb : 0);
    int zpc = 0;
    for (const Irrep& r : p.out) zpc += r.dim;
    const int units = bwd ? (int)p.instr.size() : (int)p.out.size();

    auto extra = [&](int ps) {
        const int warps = m.mulg * ps / 32;
        if (!bwd) return batch ? 2 * zb : 0;
        return ps * xb + 5 * warps * yb + (p.shared ? pad16(p.w_numel * e) : 0);
    };
    // Measured on B200: these kernels are bound by instruction issue, so the mapping that wins is the
    // one with the least per-thread overhead and the most independent groups per SM: one path
    // partition unless registers force more, and as many groups as shared memory admits.
    int xpc = 0;
    for (const Irrep& r : p.in1) xpc += r.dim;
    int best_ps = 1;
    if (!bwd) {
        auto regs = [&](int ps) { return zpc * m.nch / ps + xpc * m.nch + std::min(p.y_dim, 32) + 56; };
        while (regs(best_ps) > 232 && best_ps < 4 && best_ps * 2 <= units) best_ps *= 2;
    }
    auto groups_that_fit = [&](const Mapping& base, int ps) {
        Mapping t = base;
        t.ps = ps;
        t.extra_bytes = extra(ps);
        const int g = m.mulg * ps;
        const int want = std::max(1, std::min(8, (bwd ? 512 : (g >= 128 ? 128 : 256)) / g));
        for (int cand = want; cand >= 1; --cand) {
            t.ng = cand;
            if (t.smem(cand > 1 ? 2 : (bwd ? 2 : 3)) <= SMEM_LIMIT || (cand == 1 && t.smem(2) <= SMEM_LIMIT)) return cand;
        }
        return 0;
    };
    m.phase_of_instr.assign(p.instr.size(), 0);
    int best_ng = groups_that_fit(m, best_ps);
    m.nph = 1;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    const int max_phases = env_int("OEQ_B200_PHASES", 2);
    if (bwd && !batch && !p.shared) {
        // One or two groups per SM leave the issue slots half empty.  Stage the output-gradient row (the
        // bulk of a backward stage) in slices: cut the output irreps into nph runs of about equal width at
        // boundaries where the weights (ordered by instruction) split the same way; keep the largest
        // group count, preferring fewer phases.
        // (measured: going from one group to two pays; slicing further to reach three or four does not)
        const int target_groups = std::max(1, std::min(env_int("OEQ_B200_PHASE_GROUPS", 2), 512 / (m.mulg * best_ps)));
        for (int nph = 2; nph <= max_phases && best_ng < target_groups; ++nph) {
            std::vector<int> cut = {0};          // output irrep index where each phase starts
            for (int q = 1; q < nph; ++q) {
                const int want = (int)((long long)p.z_dim * q / nph);
                int best = -1;
                for (size_t os = cut.back() + 1; os < p.out.size(); ++os)
                    if (best < 0 || std::abs(p.out[os].off - want) < std::abs(p.out[best].off - want)) best = (int)os;
                if (best < 0) break;
                cut.push_back(best);
            }
            if ((int)cut.size() != nph) continue;
            cut.push_back((int)p.out.size());
            std::vector<int> zb(nph + 1), wbeg(nph + 1);
            bool ok = true;
            for (int q = 0; q <= nph; ++q) zb[q] = q == nph ? p.z_dim : p.out[cut[q]].off;
            // weights of phase q must be the contiguous run [wbeg[q], wbeg[q+1])
            wbeg[0] = 0;
            wbeg[nph] = p.w_numel;
            for (int q = 1; q < nph && ok; ++q) {
                int lo = p.w_numel;
                for (const Instr& t : p.instr)
                    if (t.io >= cut[q]) lo = std::min(lo, t.w_off);
                wbeg[q] = lo;
            }
            std::vector<int> phase(p.instr.size(), 0);
            for (size_t i = 0; i < p.instr.size() && ok; ++i) {
                const Instr& t = p.instr[i];
                int q = 0;
                while (q + 1 < nph && t.io >= cut[q + 1]) ++q;
                phase[i] = q;
                const int size = p.in1[t.i1].mul * p.in2[t.i2].mul;
                if (t.w_off < wbeg[q] || t.w_off + size > wbeg[q + 1]) ok = false;
            }
            for (int q = 0; q <= nph && ok; ++q)
                if ((zb[q] * e) % 16 || (wbeg[q] * e) % 16) ok = false;
            for (int q = 0; q < nph && ok; ++q)
                if (zb[q + 1] <= zb[q] || wbeg[q + 1] <= wbeg[q]) ok = false;
            if (!ok) continue;
            int wmax = 0, zmax = 0;
            for (int q = 0; q < nph; ++q) {
                wmax = std::max(wmax, wbeg[q + 1] - wbeg[q]);
                zmax = std::max(zmax, zb[q + 1] - zb[q]);
            }
            Mapping t = m;
            t.stage_bytes = xb + yb + (p.unit ? 0 : pad16(wmax * e)) + pad16(zmax * e);
            const int ng = groups_that_fit(t, best_ps);
            if (ng > best_ng) {
                best_ng = ng;
                m.stage_bytes = t.stage_bytes;
                m.nph = nph;
                m.z_ph_begin = zb;
                m.w_ph_begin = wbeg;
                m.phase_of_instr = phase;
            }
        }
    }
    if (best_ng == 0)
        return fail(OEQ_ERR_UNSUPPORTED, "problem rows do not fit in shared memory (two stages of one item exceed 227 KB)");
    m.ps = env_int(bwd ? "OEQ_B200_PS_BWD" : "OEQ_B200_PS_FWD", env_int("OEQ_B200_PS", best_ps));
    m.ng = env_int(bwd ? "OEQ_B200_NG_BWD" : "OEQ_B200_NG_FWD", env_int("OEQ_B200_NG", best_ng));
    m.extra_bytes = extra(m.ps);
    // a dedicated staging warp pays off for one wide group per CTA; many narrow groups stage their own items
    m.producer = env_int("OEQ_B200_PRODUCER", (m.ng <= 4 && m.mulg * m.ps >= 128) ? 1 : 0);
    if (m.ng > 4) m.producer = 0;
    {
        // let the compiler budget registers for as many CTAs per SM as shared memory admits
        const int stages = std::min(m.max_stages(), env_int("OEQ_B200_STAGES", 4));
        const int by_smem = stages >= 2 ? SMEM_LIMIT / (m.smem(stages) + 1024) : 1;
        const int by_threads = 2048 / m.threads();
        m.min_ctas = env_int("OEQ_B200_MIN_CTAS", std::max(1, std::min({by_smem, by_threads, 2})));
    }
    if (m.smem(2) > SMEM_LIMIT || m.ng * m.mulg * m.ps > 992 || m.ng < 1 || m.ng > 8)
        return fail(OEQ_ERR_INVALID, "OEQ_B200_PS / OEQ_B200_NG override does not fit");
    if (!bwd && !batch) apply_edges_per_item(p, m, m.extra_bytes);
    // deterministic walks align every chunk at a segment boundary (two dependent index reads per chunk)
    m.chunk_floor = (kind == K_FWD_DET || kind == K_BWD_DET) ? 64 : 32;
    assign_partitions(p, bwd, m);
    if (env_int("OEQ_B200_VERBOSE", 0))
        fprintf(stderr, "[oeq_b200] kind %d: mulg %d nch %d ps %d ng %d threads %d stage %d B extra %d B max stages %d\n",
                kind, m.mulg, m.nch, m.ps, m.ng, m.threads(), m.stage_bytes, m.extra_bytes, m.max_stages());
    return OEQ_OK;
}

// Receiver-order backward pass of the convolution (uvu_kernels.cuh, run_backward_recv): one thread per
// channel, stages as in the forward pass, two dX rows and the dY partials per group as extras.
constexpr int K_BWD_RECV_DET = 6, K_BWD_RECV_ATOMIC = 7;

bool recv_backward_supported(const Problem& p) {
    if (p.mode != OEQ_MODE_UVU || p.shared || p.y_dim > 32) return false;
    for (const Irrep& r : p.in2)
        if (r.mul != 1) return false;
    int maxmul = 1, zpc = 0, xpc = 0;
    for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
    for (const Irrep& r : p.out) { maxmul = std::max(maxmul, r.mul); zpc += r.dim; }
    for (const Irrep& r : p.in1) xpc += r.dim;
    if (maxmul > 256) return false;                             // one thread per channel
    int d1max = 1;
    for (const Irrep& r : p.in1) d1max = std::max(d1max, r.dim);
    // the channel's slice of dZ lives in registers (32-bit registers: twice as many for FP64 values)
    if ((zpc + 2 * p.y_dim + 4 * d1max) * (p.elem() / 4) + 40 > 200) return false;
    return env_int("OEQ_B200_BWD_RECV", 1) != 0;
}

int choose_mapping_recv(const Problem& p, Mapping& m) {
    int maxmul = 1;
    for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
    for (const Irrep& r : p.out) maxmul = std::max(maxmul, r.mul);
    m.mulg = (maxmul + 31) / 32 * 32;
    m.nch = 1;
    m.ps = 1;
    const int e = p.elem();
    const int xb = pad16(p.x_dim * e), yb = pad16(p.y_dim * e), wb = p.unit ? 0 : pad16(p.w_numel * e);
    m.sw_bytes = 0;
    m.stage_bytes = xb + yb + wb;
    // dZ values per channel beyond the register budget are parked in shared memory (whole output irreps)
    int zpc = 0;
    for (const Irrep& r : p.out) zpc += r.dim;
    const int budget = env_int("OEQ_B200_GZ_REGS", p.dtype == OEQ_F64 ? 28 : 56);
    m.gz_regs = budget;
    m.gz_smem_values = 0;
    {
        int off = 0;
        for (const Irrep& r : p.out) {
            if (off >= budget) m.gz_smem_values += r.dim;
            off += r.dim;
        }
    }
    m.extra_bytes = 2 * xb + 5 * (m.mulg / 32) * yb + pad16(m.gz_smem_values * m.mulg * e);
    m.nph = 1;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    // two wide groups share a CTA (one CTA per SM): 320 threads leave 200 registers per thread, which the
    // channel's dZ slice needs; two CTAs of 160 threads would be capped at 168
    const int want = std::max(1, std::min(8, 256 / m.mulg));
    m.ng = 0;
    for (int cand = want; cand >= 1 && !m.ng; --cand) {
        m.ng = cand;
        if (m.smem(cand > 1 ? 2 : 3) > SMEM_LIMIT && !(cand == 1 && m.smem(2) <= SMEM_LIMIT)) m.ng = 0;
    }
    if (!m.ng) return fail(OEQ_ERR_UNSUPPORTED, "problem rows do not fit in shared memory");
    m.ng = env_int("OEQ_B200_NG_RECV", m.ng);
    m.producer = env_int("OEQ_B200_PRODUCER", (m.ng <= 4 && m.mulg >= 128) ? 1 : 0);
    if (m.ng > 4) m.producer = 0;
    const int stages = std::min(m.max_stages(), env_int("OEQ_B200_STAGES", 4));
    const int by_smem = stages >= 2 ? SMEM_LIMIT / (m.smem(stages) + 1024) : 1;
    const int by_threads = 2048 / m.threads();
    m.min_ctas = env_int("OEQ_B200_MIN_CTAS_RECV", std::max(1, std::min({by_smem, by_threads, 2})));
    if (m.smem(2) > SMEM_LIMIT || m.ng < 1 || m.ng > 8) return fail(OEQ_ERR_INVALID, "OEQ_B200_NG_RECV override does not fit");
    apply_edges_per_item(p, m, m.extra_bytes);
    assign_partitions(p, true, m);
    if (env_int("OEQ_B200_VERBOSE", 0))
        fprintf(stderr, "[oeq_b200] receiver-order backward: mulg %d ng %d threads %d stage %d B extra %d B max stages %d min ctas %d\n",
                m.mulg, m.ng, m.threads(), m.stage_bytes, m.extra_bytes, m.max_stages(), m.min_ctas);
    return OEQ_OK;
}

// ------------------------------------------------------------------ descriptor text

template <class V, class F>
void emit_array(std::ostringstream& s, const char* type, const char* name, const V& v, F&& fmt) {
    s << "constexpr " << type << " " << name << "[] = {";
    if (v.empty()) s << "0";
    for (size_t i = 0; i < v.size(); ++i) {
        if (i) s << ", ";
        fmt(s, v[i]);
    }
    s << "};\n";
}

struct UvwConfig {
    int tile_r = 16, uvc = 64, dmax = 1, mwmax = 1, threads = 256;
    int smem(const Problem& p, bool bwd) const {
        auto r4 = [](long long n) { return (n + 3) / 4 * 4; };
        long long e = r4((long long)tile_r * p.x_dim) + r4((long long)tile_r * p.y_dim) + r4((long long)tile_r * p.z_dim) +
                      r4((long long)uvc * tile_r * dmax);
        if (bwd)
            e += r4((long long)tile_r * p.x_dim) + r4((long long)tile_r * p.y_dim) + r4((long long)mwmax * tile_r * dmax) +
                 r4((long long)uvc * tile_r * dmax);
        return (int)std::min<long long>(e * p.elem(), 1ll << 30);
    }
};

int choose_uvw(const Problem& p, bool bwd, UvwConfig& c) {
    for (const Irrep& r : p.out) {
        c.dmax = std::max(c.dmax, r.dim);
        c.mwmax = std::max(c.mwmax, r.mul);
    }
    int max_uv = 1;
    for (const Instr& t : p.instr) max_uv = std::max(max_uv, p.in1[t.i1].mul * p.in2[t.i2].mul);
    c.uvc = std::min(64, max_uv);
    for (int tile : {16, 8, 4}) {
        c.tile_r = tile;
        if (c.smem(p, bwd) <= SMEM_LIMIT) return OEQ_OK;
    }
    return fail(OEQ_ERR_UNSUPPORTED, "'uvw' problem rows do not fit in shared memory");
}

// ---- tensor-core forward pass of the 'uvu' convolution (mirrors the constexpr geometry of uvu_tc_kernels.cuh)
// Entry e of the per-edge matrix M[(p,k)][i] = sum_j c^p_ijk y_j: where it lives in the swizzled B tile and
// which (j, coefficient) terms it sums (dense [entry][tmax] table, coefficient 0 where an entry has fewer).
struct UvuTcTables {
    int n = 0, tmax = 1;
    std::vector<int> off, term_j;
    std::vector<double> term_c;
    int xpc = 0;
};

// Columns of the per-edge product: the paths of consumer partition q (the partition of their output
// irrep) are contiguous, in instruction order, and start at a multiple of 16.
struct UvuTcColumns {
    std::vector<int> col_begin;   // per instruction
    std::vector<int> part_col;    // per partition, plus the padded total
};

UvuTcColumns uvu_tc_columns(const Problem& p, const std::vector<int>& part_of_out, int parts) {
    UvuTcColumns c;
    c.col_begin.assign(p.instr.size(), 0);
    int cur = 0;
    for (int q = 0; q < parts; ++q) {
        cur = (cur + 15) / 16 * 16;
        c.part_col.push_back(cur);
        for (size_t i = 0; i < p.instr.size(); ++i)
            if (part_of_out[p.instr[i].io] == q) {
                c.col_begin[i] = cur;
                cur += p.out[p.instr[i].io].dim;
            }
    }
    c.part_col.push_back((cur + 15) / 16 * 16);
    return c;
}

int tc_swizzle_host(int row, int col) {
    return (row >> 3) * 1024 + (row & 7) * 128 + ((((col >> 2) ^ (row & 7)) & 7) << 4) + ((col & 3) << 2);
}

UvuTcTables build_uvu_tc_tables(const Problem& p, const UvuTcColumns& cols) {
    UvuTcTables t;
    std::vector<int> xoff(p.in1.size(), 0);
    for (size_t a = 0; a < p.in1.size(); ++a) {
        xoff[a] = t.xpc;
        t.xpc += p.in1[a].dim;
    }
    std::vector<std::vector<std::pair<int, double>>> terms;
    for (size_t pi = 0; pi < p.instr.size(); ++pi) {
        const Instr& ins = p.instr[pi];
        const int col0 = cols.col_begin[pi];
        const int d1 = p.in1[ins.i1].dim, d3 = p.out[ins.io].dim;
        for (int k = 0; k < d3; ++k)
            for (int i = 0; i < d1; ++i) {
                std::vector<std::pair<int, double>> tt;
                for (size_t z = 0; z < ins.ci.size(); ++z)
                    if (ins.ci[z] == i && ins.ck[z] == k) tt.push_back({p.in2[ins.i2].off + ins.cj[z], ins.cv[z]});
                if (tt.empty()) continue;
                t.off.push_back(tc_swizzle_host(col0 + k, xoff[ins.i1] + i));
                t.tmax = std::max(t.tmax, (int)tt.size());
                terms.push_back(std::move(tt));
            }
    }
    t.n = (int)t.off.size();
    t.term_j.assign((size_t)std::max(1, t.n) * t.tmax, 0);
    t.term_c.assign((size_t)std::max(1, t.n) * t.tmax, 0.0);
    for (int e = 0; e < t.n; ++e)
        for (size_t z = 0; z < terms[e].size(); ++z) {
            t.term_j[(size_t)e * t.tmax + z] = terms[e][z].first;
            t.term_c[(size_t)e * t.tmax + z] = terms[e][z].second;
        }
    if (t.off.empty()) t.off.push_back(0);
    return t;
}

struct UvuTcGeometry {
    int stages = 0, smem = 0;
};

// Problems the tensor-core forward pass takes: FP32 'uvu' with per-edge weights, second input of
// multiplicity 1 and at most 32 components, widest multiplicity 65..128 (thread = channel, M = 128 rows),
// at most 32 first-input components per channel (one swizzled 128-byte row) and 256 output columns.
bool uvu_tc_geometry(const Problem& p, UvuTcGeometry& g, int npad = 0) {
    if (p.mode != OEQ_MODE_UVU || p.shared || p.unit || p.dtype != OEQ_F32) return false;
    // Opt-in: measured on B200 the per-edge hand-offs between the roles make this kernel about twice as slow
    // as the FMA kernel (MACE-large, 1.5 M edges: 14.0 ms against 7.2 ms), so the FMA kernel is the default.
    if (!env_int("OEQ_B200_UVU_TC", 0)) return false;
    if (p.y_dim > 32) return false;
    int maxmul = 0, xpc = 0, ncols = 0;
    for (const Irrep& r : p.in1) {
        maxmul = std::max(maxmul, r.mul);
        xpc += r.dim;
    }
    for (const Instr& t : p.instr) {
        if (p.in2[t.i2].mul != 1) return false;
        ncols += p.out[t.io].dim;
    }
    if (maxmul <= 64 || maxmul > 128 || xpc > 32 || ncols > 224 || ncols == 0) return false;
    if ((p.x_dim * 4) % 16 || (p.w_numel * 4) % 16) return false;
    if (npad == 0) npad = (ncols + 15) / 16 * 16 + 16;      // upper bound: one padding gap between two partitions
    if (npad > 256) return false;
    const int off_stage = 2 * 2 * 128 * 128 + 2 * 2 * npad * 128 + 512;
    const int stage = pad16(p.x_dim * 4) + pad16(p.w_numel * 4) + pad16(p.y_dim * 4);
    g.stages = std::min(4, (SMEM_LIMIT - 1024 - off_stage) / stage);
    if (g.stages < 3) return false;
    g.smem = 1024 + off_stage + g.stages * stage;
    return true;
}

// Tables of the slice kernels: the paths grouped by their two input irreps (first-input major), and the
// Clebsch-Gordan entries of a group ordered by (i, j), so that a product x_i y_j is formed once for all its paths.
void emit_slice_tables(std::ostringstream& s, const Problem& p, const Mapping& m) {
    struct Entry { int i, j, path, k, n; double v; };
    std::vector<int> ga, gb, g0 = {0}, pri, prj, ge = {0}, gp = {0}, plist, toff(p.instr.size(), 0), ei, ej, et, enew, efirst;
    std::vector<std::vector<int>> pr(p.instr.size());       // the products of a path's coefficients
    std::vector<double> ev;
    int tmax = 1;
    for (size_t a = 0; a < p.in1.size(); ++a)
        for (size_t b = 0; b < p.in2.size(); ++b) {
            std::vector<Entry> es;
            int t = 0;
            for (size_t q = 0; q < p.instr.size(); ++q) {
                const Instr& ins = p.instr[q];
                if (ins.i1 != (int)a || ins.i2 != (int)b) continue;
                plist.push_back((int)q);
                toff[q] = t;
                t += p.out[ins.io].dim;
                for (size_t z = 0; z < ins.cv.size(); ++z) es.push_back({ins.ci[z], ins.cj[z], (int)q, ins.ck[z], (int)z, ins.cv[z]});
                pr[q].assign(ins.cv.size(), 0);
            }
            if (t == 0) continue;
            tmax = std::max(tmax, t);
            std::stable_sort(es.begin(), es.end(), [](const Entry& x, const Entry& y) {
                return std::make_tuple(x.i, x.j, x.path, x.k) < std::make_tuple(y.i, y.j, y.path, y.k);
            });
            std::vector<int> seen(t, 0);
            for (size_t n = 0; n < es.size(); ++n) {
                const int tt = toff[es[n].path] + es[n].k;
                ei.push_back(es[n].i); ej.push_back(es[n].j); et.push_back(tt); ev.push_back(es[n].v);
                enew.push_back(n == 0 || es[n].i != es[n - 1].i || es[n].j != es[n - 1].j);
                if (enew.back()) { pri.push_back(es[n].i); prj.push_back(es[n].j); }
                pr[es[n].path][es[n].n] = (int)pri.size() - 1;
                efirst.push_back(!seen[tt]);
                seen[tt] = 1;
            }
            ga.push_back((int)a); gb.push_back((int)b); g0.push_back((int)pri.size());
            ge.push_back((int)ei.size()); gp.push_back((int)plist.size());
        }
    auto put_int = [](std::ostringstream& o, int v) { o << v; };
    s << "constexpr int NSLICE = " << m.n_slice << ", SLICE_WARPS = " << m.slice_warps << ", SLICE_STAGES = " << m.slice_stages << ", SLICE_CPL = " << m.slice_cpl << ", SLICE_ONE = " << (m.slice_one ? 1 : 0)
      << ", N_GROUPS = " << ga.size() << ", T_MAX = " << tmax << ", N_OUTER = " << pri.size() << ";\n";
    s << "constexpr bool SLICE_FULL = " << (m.slice_full ? "true" : "false") << ", SLICE_OUTER = " << (m.slice_outer ? "true" : "false") << ";\n";
    std::vector<int> cgpr;
    for (const std::vector<int>& v : pr) cgpr.insert(cgpr.end(), v.begin(), v.end());
    emit_array(s, "int", "GRP_PR", g0, put_int);
    emit_array(s, "int", "PR_I", pri, put_int);
    emit_array(s, "int", "PR_J", prj, put_int);
    emit_array(s, "int", "CG_PR", cgpr, put_int);
    emit_array(s, "int", "GRP_A", ga, put_int);
    emit_array(s, "int", "GRP_B", gb, put_int);
    emit_array(s, "int", "GRP_E", ge, put_int);
    emit_array(s, "int", "GRP_P", gp, put_int);
    emit_array(s, "int", "P_LIST", plist, put_int);
    emit_array(s, "int", "T_OFF", toff, put_int);
    emit_array(s, "int", "E_I", ei, put_int);
    emit_array(s, "int", "E_J", ej, put_int);
    emit_array(s, "int", "E_T", et, put_int);
    emit_array(s, "bool", "E_NEW", enew, put_int);
    emit_array(s, "bool", "E_FIRST", efirst, put_int);
    const bool f64 = p.dtype == OEQ_F64;
    emit_array(s, "T", "E_V", ev, [f64](std::ostringstream& o, double v) {
        char buf[64];
        if (f64) snprintf(buf, sizeof buf, "%a", v);
        else snprintf(buf, sizeof buf, "%af", (double)(float)v);
        o << buf;
    });
}

std::string descriptor_text(const Problem& p, const Mapping& m, const UvwConfig* uvw = nullptr) {
    std::ostringstream s;
    s.precision(17);
    s << "// problem descriptor (tables only; kernel bodies are in the included headers)\n";
    s << "namespace oeqd {\n";
    s << "typedef " << (p.dtype == OEQ_F64 ? "double" : "float") << " T;\n";
    s << "constexpr int X_DIM = " << p.x_dim << ", Y_DIM = " << p.y_dim << ", Z_DIM = " << p.z_dim
      << ", W_NUMEL = " << p.w_numel << ";\n";
    s << "constexpr bool SHARED_W = " << (p.shared ? "true" : "false") << ";\n";
    if (p.mode == OEQ_MODE_UVW) {
        auto put = [](std::ostringstream& o, int v) { o << v; };
        std::vector<int> begin = {0}, start, mul, off;
        for (size_t n = 0; n < p.instr.size(); ++n) {
            if (n < p.subs.size())
                for (const Problem::Sub& q : p.subs[n]) { start.push_back(q.start); mul.push_back(q.mul); off.push_back(q.w_off); }
            begin.push_back((int)start.size());
        }
        emit_array(s, "int", "SUB_BEGIN", begin, put);
        emit_array(s, "int", "SUB_START", start, put);
        emit_array(s, "int", "SUB_MUL", mul, put);
        emit_array(s, "int", "SUB_WOFF", off, put);
    }
    s << "constexpr bool UNIT_Y = " << (p.unit_y ? "true" : "false") << ", TRANSPOSED_W = " << (p.transposed_w ? "true" : "false") << ";\n";
    s << "constexpr bool UNIT_W = " << (p.unit ? "true" : "false") << ";\n";
    s << "constexpr int N_IN1 = " << p.in1.size() << ", N_IN2 = " << p.in2.size() << ", N_OUT = " << p.out.size()
      << ", N_INSTR = " << p.instr.size() << ";\n";
    auto put_int = [](std::ostringstream& o, int v) { o << v; };
    auto irreps = [&](const char* prefix, const std::vector<Irrep>& v) {
        std::vector<int> mul, dim, off;
        for (const Irrep& r : v) {
            mul.push_back(r.mul); dim.push_back(r.dim); off.push_back(r.off);
        }
        emit_array(s, "int", (std::string(prefix) + "_MUL").c_str(), mul, put_int);
        emit_array(s, "int", (std::string(prefix) + "_D").c_str(), dim, put_int);
        emit_array(s, "int", (std::string(prefix) + "_OFF").c_str(), off, put_int);
    };
    irreps("IN1", p.in1);
    irreps("IN2", p.in2);
    irreps("OUT", p.out);
    std::vector<int> i1, i2, io, woff, begin, ci, cj, ck;
    std::vector<double> cv;
    for (const Instr& t : p.instr) {
        i1.push_back(t.i1); i2.push_back(t.i2); io.push_back(t.io); woff.push_back(t.w_off);
        begin.push_back((int)ci.size());
        ci.insert(ci.end(), t.ci.begin(), t.ci.end());
        cj.insert(cj.end(), t.cj.begin(), t.cj.end());
        ck.insert(ck.end(), t.ck.begin(), t.ck.end());
        cv.insert(cv.end(), t.cv.begin(), t.cv.end());
    }
    begin.push_back((int)ci.size());
    emit_array(s, "int", "I_IN1", i1, put_int);
    emit_array(s, "int", "I_IN2", i2, put_int);
    emit_array(s, "int", "I_OUT", io, put_int);
    emit_array(s, "int", "W_OFF", woff, put_int);
    emit_array(s, "int", "CG_BEGIN", begin, put_int);
    emit_array(s, "int", "CG_I", ci, put_int);
    emit_array(s, "int", "CG_J", cj, put_int);
    emit_array(s, "int", "CG_K", ck, put_int);
    const bool f64 = p.dtype == OEQ_F64;
    emit_array(s, "T", "CG_V", cv, [f64](std::ostringstream& o, double v) {
        char buf[64];
        if (f64) snprintf(buf, sizeof buf, "%a", v);
        else snprintf(buf, sizeof buf, "%af", (double)(float)v);
        o << buf;
    });
    s << "constexpr int MULG = " << m.mulg << ", NCH = " << m.nch << ", PS = " << m.ps << ", NG = " << m.ng
      << ", PRODUCER = " << m.producer << ", MIN_CTAS = " << m.min_ctas << ", EPI = " << m.epi << ";\n";
    emit_array(s, "int", "FWD_PART_OF_OUT", m.part_of_out, put_int);
    emit_array(s, "int", "BWD_PART_OF_INSTR", m.part_of_instr, put_int);
    emit_array(s, "int", "ZR_OFF", m.zr_off, put_int);
    emit_array(s, "int", "XR_OFF", m.xr_off, put_int);
    {
        std::vector<int> ph = m.phase_of_instr;
        ph.resize(p.instr.size(), 0);
        emit_array(s, "int", "BWD_PHASE_OF_INSTR", ph, put_int);
        s << "constexpr int BWD_NPH = " << m.nph << ";\n";
        std::vector<int> zb = m.z_ph_begin, wb2 = m.w_ph_begin;
        if (zb.empty()) zb = {0, p.z_dim};
        if (wb2.empty()) wb2 = {0, p.w_numel};
        emit_array(s, "int", "Z_PH_BEGIN", zb, put_int);
        emit_array(s, "int", "W_PH_BEGIN", wb2, put_int);
        // the same tables again with device storage, for run-time indexing by phase
        s << "__device__ const int Z_PH_BEGIN_DEV[] = {";
        for (size_t i = 0; i < zb.size(); ++i) s << (i ? ", " : "") << zb[i];
        s << "};\n__device__ const int W_PH_BEGIN_DEV[] = {";
        for (size_t i = 0; i < wb2.size(); ++i) s << (i ? ", " : "") << wb2[i];
        s << "};\n";
    }
    s << "constexpr int ZPC_MAX = " << m.zpc_max << ", XPC = " << m.xpc << ";\n";
    s << "constexpr int GZ_REGS = " << m.gz_regs << ", GZ_SMEM_VALUES = " << m.gz_smem_values << ";\n";
    // cycle accounting inside the kernels is a development aid: it exists only in a library built with
    // -DOEQ_DEV_PROFILE (the shipped entry points then contain no allocation, synchronisation or printing)
#ifdef OEQ_DEV_PROFILE
    s << "constexpr bool UVU_PROFILE = " << (env_int("OEQ_B200_UVU_PROFILE", 0) ? "true" : "false") << ";\n";
#else
    s << "constexpr bool UVU_PROFILE = false;\n";
#endif
    if (m.tc_tables) {
        const UvuTcColumns cols = uvu_tc_columns(p, m.part_of_out, m.ps);
        const UvuTcTables t = build_uvu_tc_tables(p, cols);
        emit_array(s, "int", "TC_COL_BEGIN", cols.col_begin, put_int);
        emit_array(s, "int", "TC_PART_COL", cols.part_col, put_int);
        s << "constexpr int TCM_N = " << t.n << ", TCM_TMAX = " << t.tmax << ";\n";
        auto dev_ints = [&](const char* name, const std::vector<int>& v) {
            s << "__device__ const int " << name << "[] = {";
            for (size_t i = 0; i < v.size(); ++i) s << (i ? ", " : "") << v[i];
            s << "};\n";
        };
        dev_ints("TCM_OFF_DEV", t.off);
        dev_ints("TCM_J_DEV", t.term_j);
        s << "__device__ const float TCM_C_DEV[] = {";
        for (size_t i = 0; i < t.term_c.size(); ++i) {
            char buf[64];
            snprintf(buf, sizeof buf, "%af", (double)(float)t.term_c[i]);
            s << (i ? ", " : "") << buf;
        }
        s << "};\n";
    }
    if (m.slice_warps) emit_slice_tables(s, p, m);
    if (uvw)
        s << "constexpr int TILE_R = " << uvw->tile_r << ", UVC = " << uvw->uvc << ", DMAX = " << uvw->dmax
          << ", MWMAX = " << uvw->mwmax << ", UVW_THREADS = " << uvw->threads << ";\n";
    s << "}  // namespace oeqd\n";
    return s.str();
}

// ------------------------------------------------------------------ compile + cache

unsigned long long fnv1a(const std::string& s, unsigned long long h = 1469598103934665603ull) {
    for (unsigned char c : s) {
        h ^= c;
        h *= 1099511628211ull;
    }
    return h;
}

bool read_file(const std::string& path, std::string& out) {
    std::ifstream f(path, std::ios::binary);
    if (!f) return false;
    std::ostringstream ss;
    ss << f.rdbuf();
    out = ss.str();
    return true;
}

struct Compiled {
    std::string cubin;
    std::string log;
};

int compile_kernel(const std::string& descriptor, const std::string& main_header, int kernel_id, Compiled& out) {
    std::lock_guard<std::mutex> lock(g_mutex);
    const std::string dir = kernel_dir();
    std::string common, body;
    if (!read_file(dir + "/oeq_common.cuh", common) || !read_file(dir + "/" + main_header, body))
        return fail(OEQ_ERR_COMPILE, "kernel headers not found in " + dir);
    for (const char* inc : {"tc_common.cuh", "uvw_ts_common.cuh", "uvu_kernels.cuh", "uvw_kernels.cuh"}) {   // headers that the kernel files include
        std::string text;
        if (main_header != inc && read_file(dir + "/" + inc, text)) common += text;
    }
    const std::string source = descriptor + "#define OEQ_KERNEL " + std::to_string(kernel_id) + "\n#include \"" +
                               main_header + "\"\n";
    const std::string options = "-arch=sm_100a -std=c++17 -lineinfo -default-device -diag-suppress 177";
    unsigned long long h = fnv1a(source);
    h = fnv1a(common, h);
    h = fnv1a(body, h);
    h = fnv1a(options, h);
    char name[64];
    snprintf(name, sizeof name, "/k_%016llx.cubin", h);
    const std::string cdir = cache_dir();
    const std::string path = cdir + name;
    if (!env_int("OEQ_B200_NO_CACHE", 0) && read_file(path, out.cubin) && !out.cubin.empty()) return OEQ_OK;

    int rc = load_nvrtc();
    if (rc) return rc;
    nvrtcProgram prog;
    if (g_nvrtc.create(&prog, source.c_str(), "oeq_specialisation.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        return fail(OEQ_ERR_COMPILE, "nvrtcCreateProgram failed");
    const std::string inc = "-I" + dir;
    std::vector<const char*> opts = {"-arch=sm_100a", "-std=c++17", "-lineinfo", "-default-device", "-diag-suppress=177", inc.c_str()};
    std::string ptxas_v = "--ptxas-options=-v";
    if (env_int("OEQ_B200_VERBOSE", 0)) opts.push_back(ptxas_v.c_str());
    std::string maxreg = "--maxrregcount=" + std::to_string(env_int("OEQ_B200_MAXRREG", 0));
    if (env_int("OEQ_B200_MAXRREG", 0) > 0) opts.push_back(maxreg.c_str());
    nvrtcResult res = g_nvrtc.compile(prog, (int)opts.size(), opts.data());
    size_t log_size = 0;
    g_nvrtc.log_size(prog, &log_size);
    out.log.assign(log_size, '\0');
    if (log_size > 1) g_nvrtc.log(prog, &out.log[0]);
    if (env_int("OEQ_B200_VERBOSE", 0) && log_size > 1) fprintf(stderr, "[oeq_b200] %s\n", out.log.c_str());
    if (res != NVRTC_SUCCESS) {
        g_nvrtc.destroy(&prog);
        if (env_int("OEQ_B200_KEEP_SOURCE", 0)) {
            std::ofstream f("/tmp/oeq_failed_specialisation.cu");
            f << source;
        }
        return fail(OEQ_ERR_COMPILE, std::string("kernel specialisation failed: ") + g_nvrtc.error_string(res) + "\n" +
                                         out.log.substr(0, 4000));
    }
    size_t size = 0;
    g_nvrtc.cubin_size(prog, &size);
    out.cubin.assign(size, '\0');
    g_nvrtc.cubin(prog, &out.cubin[0]);
    g_nvrtc.destroy(&prog);
    mkdir(cdir.c_str(), 0755);
    const std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
    {
        std::ofstream f(tmp, std::ios::binary);
        f.write(out.cubin.data(), (std::streamsize)out.cubin.size());
    }
    rename(tmp.c_str(), path.c_str());
    return OEQ_OK;
}

// ------------------------------------------------------------------ a specialised kernel

struct Kernel {
    Mapping map;
    UvwConfig uvw;
    bool is_uvw = false, is_uvw_row = false;
    int row_smem = 0;             // is_uvw_row: shared memory of a CTA
    Compiled code;
    bool compiled = false, loaded = false;
    cudaLibrary_t lib = nullptr;
    cudaKernel_t fn = nullptr, reduce_fn = nullptr;
    int stages = 0, smem = 0, regs = 0, ctas_per_sm = 1, sm_count = 0;
    bool is_uvu_tc = false;       // tensor-core forward of the convolution: one CTA per SM
    UvuTcGeometry tc_geo;
    int threads() const { return map.slice_warps ? 32 * map.slice_warps : (is_uvu_tc ? 128 * map.ps + 64 : map.threads()); }
};

int build_uvu(const Problem& p, int kind, Kernel& k) {
    int rc = choose_mapping(p, kind, k.map);
    if (rc) return rc;
    rc = compile_kernel(descriptor_text(p, k.map), "uvu_kernels.cuh", kind, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// One-pass second derivatives of the batch 'uvu' product (uvu_kernels.cuh, run_double_backward): per-row
// weights, second input of multiplicity 1 with at most 32 components, at most 256 channels; a row's seven
// arrays form one stage.
constexpr int K_DBL_BATCH = 8;

bool double_backward_supported(const Problem& p) {
    if (p.mode != OEQ_MODE_UVU || p.shared || p.unit || p.y_dim > 32) return false;
    for (const Irrep& r : p.in2)
        if (r.mul != 1) return false;
    int maxmul = 1, zpc = 0, d1max = 1;
    for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
    for (const Irrep& r : p.out) { maxmul = std::max(maxmul, r.mul); zpc += r.dim; }
    for (const Irrep& r : p.in1) d1max = std::max(d1max, r.dim);
    if (maxmul > 256) return false;
    if ((zpc + 3 * p.y_dim + 5 * d1max) * (p.elem() / 4) + 40 > 232) return false;   // registers per thread
    return env_int("OEQ_B200_FUSED_DOUBLE_BACKWARD", 1) != 0;
}

int build_uvu_dbl(const Problem& p, Kernel& k) {
    Mapping& m = k.map;
    int maxmul = 1;
    for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
    for (const Irrep& r : p.out) maxmul = std::max(maxmul, r.mul);
    m.mulg = (maxmul + 31) / 32 * 32;
    m.nch = 1; m.ps = 1; m.producer = 1;
    const int e = p.elem();
    const int xb = pad16(p.x_dim * e), yb = pad16(p.y_dim * e), wb = pad16(p.w_numel * e), zb = pad16(p.z_dim * e);
    m.sw_bytes = 0;
    m.stage_bytes = 2 * xb + 2 * yb + 2 * wb + zb;
    m.extra_bytes = 5 * (m.mulg / 32) * yb;
    m.nph = 1;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    m.ng = 0;
    for (int cand = std::max(1, std::min(4, 256 / m.mulg)); cand >= 1 && !m.ng; --cand) {
        m.ng = cand;
        if (m.smem(2) > SMEM_LIMIT) m.ng = 0;
    }
    if (!m.ng) return fail(OEQ_ERR_UNSUPPORTED, "a row's seven arrays do not fit two shared-memory stages");
    const int stages = std::min(m.max_stages(), 4);
    m.min_ctas = std::max(1, std::min({stages >= 2 ? SMEM_LIMIT / (m.smem(stages) + 1024) : 1, 2048 / m.threads(), 2}));
    assign_partitions(p, true, m);
    int rc = compile_kernel(descriptor_text(p, m), "uvu_kernels.cuh", K_DBL_BATCH, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

int build_uvu_recv(const Problem& p, bool deterministic, Kernel& k) {
    int rc = choose_mapping_recv(p, k.map);
    if (rc) return rc;
    // Deterministic variant: two helper warps per CTA sum the previous block's dX rows while the consumers
    // work.  With two wide groups and their staging warps that makes twelve warps, three per scheduler, the
    // same register ceiling (168) as the ten warps without helpers.
    k.map.helper_warps = deterministic ? std::max(0, env_int("OEQ_B200_HELPER_WARPS", 2)) : 0;
    // narrow problems: their launches are too short for the pipelined row sum, and the two extra warps would
    // lower the register ceiling of the one-warp groups
    if (k.map.threads() > 1024 || k.map.epi > 1) k.map.helper_warps = 0;
    k.map.chunk_floor = deterministic ? 64 : 32;
    const std::string macros = "#define OEQ_HELPER_WARPS " + std::to_string(k.map.helper_warps) + "\n";
    rc = compile_kernel(descriptor_text(p, k.map) + macros, "uvu_kernels.cuh", deterministic ? K_BWD_RECV_DET : K_BWD_RECV_ATOMIC, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// Second derivatives of the convolution in two launches (uvu_kernels.cuh, DBLC): a forward-like walk for the
// gradient with respect to dZ and a receiver-order walk for the gradients with respect to X, Y, W.  Stages
// carry the cotangent rows next to X, Y, W.
constexpr int K_DBLC_Z_DET = 40, K_DBLC_Z_ATOMIC = 41, K_DBLC_G_DET = 42, K_DBLC_G_ATOMIC = 43;

bool conv_double_backward_supported(const Problem& p) {
    if (p.unit || !recv_backward_supported(p)) return false;
    int zpc = 0, xpc = 0;
    for (const Irrep& r : p.out) zpc += r.dim;
    for (const Irrep& r : p.in1) xpc += r.dim;
    if ((zpc + 3 * xpc + 2 * p.y_dim) * (p.elem() / 4) + 48 > 240) return false;    // registers of the forward-like walk
    return env_int("OEQ_B200_FUSED_DOUBLE_BACKWARD", 1) != 0;
}

int build_uvu_dblc(const Problem& p, bool deterministic, bool grads, Kernel& k) {
    Mapping& m = k.map;
    const int e = p.elem();
    const int xb = pad16(p.x_dim * e), yb = pad16(p.y_dim * e), wb = pad16(p.w_numel * e);
    int rc;
    if (grads) {
        if ((rc = choose_mapping_recv(p, m))) return rc;
        m.epi = 1;
        m.stage_cap = 4;
        // fewer dZ values in registers than the first-derivative pass: the cotangents take their place
        const int budget = env_int("OEQ_B200_GZ_REGS_DBL", p.dtype == OEQ_F64 ? 14 : 32);
        m.gz_regs = budget;
        m.gz_smem_values = 0;
        int off = 0;
        for (const Irrep& r : p.out) {
            if (off >= budget) m.gz_smem_values += r.dim;
            off += r.dim;
        }
        m.extra_bytes = 2 * xb + 5 * (m.mulg / 32) * yb + pad16(m.gz_smem_values * m.mulg * e);
    } else {
        int maxmul = 1;
        for (const Instr& t : p.instr) maxmul = std::max(maxmul, p.in1[t.i1].mul);
        for (const Irrep& r : p.out) maxmul = std::max(maxmul, r.mul);
        m.mulg = (maxmul + 31) / 32 * 32;
        m.nch = 1; m.ps = 1;
        m.sw_bytes = 0;
        m.extra_bytes = 0;
        m.nph = 1;
        m.z_ph_begin = {0, p.z_dim};
        m.w_ph_begin = {0, p.w_numel};
        m.phase_of_instr.assign(p.instr.size(), 0);
    }
    m.helper_warps = 0;
    m.stage_bytes = 2 * (xb + yb + wb);
    m.ng = 0;
    for (int cand = std::max(1, std::min(8, 256 / m.mulg)); cand >= 1 && !m.ng; --cand) {
        m.ng = cand;
        if (m.smem(2) > SMEM_LIMIT) m.ng = 0;
    }
    if (!m.ng) return fail(OEQ_ERR_UNSUPPORTED, "an edge's rows and cotangent rows do not fit two shared-memory stages");
    m.producer = (m.ng <= 4 && m.mulg >= 128) ? 1 : 0;
    const int stages = std::min(m.max_stages(), 4);
    m.min_ctas = std::max(1, std::min({stages >= 2 ? SMEM_LIMIT / (m.smem(stages) + 1024) : 1, 2048 / m.threads(), 2}));
    assign_partitions(p, grads, m);
    const int kind = grads ? (deterministic ? K_DBLC_G_DET : K_DBLC_G_ATOMIC) : (deterministic ? K_DBLC_Z_DET : K_DBLC_Z_ATOMIC);
    const std::string macros = "#define OEQ_HELPER_WARPS 0\n";
    rc = compile_kernel(descriptor_text(p, m) + macros, "uvu_kernels.cuh", kind, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// ---- slice kernels (uvu_slice_kernels.cuh): one warp per (edges, slice of 32 channels)
constexpr int K_SLICE_FWD_DET = 50, K_SLICE_FWD_ATOMIC = 51, K_SLICE_BWD_DET = 52, K_SLICE_BWD_ATOMIC = 53;

// A row is one slice of up to 32 channels, or every multiplicity is the same multiple of 32.
bool slice_shape(const Problem& p, Mapping& m) {
    if (p.mode != OEQ_MODE_UVU || p.shared || p.y_dim > 32) return false;
    for (const Irrep& r : p.in2)
        if (r.mul != 1) return false;
    int lo = 1 << 30, hi = 0;
    for (const Irrep& r : p.in1) { lo = std::min(lo, r.mul); hi = std::max(hi, r.mul); }
    for (const Irrep& r : p.out) { lo = std::min(lo, r.mul); hi = std::max(hi, r.mul); }
    if (hi > 256 || hi < 1) return false;
    m.slice_full = lo == hi && hi % 32 == 0;
    if (hi > 32 && !m.slice_full) return false;
    m.n_slice = m.slice_full ? hi / 32 : 1;
    return env_int("OEQ_B200_SLICE", 1) != 0;
}

// Warps per SM by the registers a thread needs (65 536 over the warps, in steps of the warps that share a
// scheduler), stages by shared memory.  `room`: registers to leave room for, where the estimate falls short.
bool slice_fit(const Problem& p, Mapping& m, int regs, int warp_bytes, int cta_bytes, bool second = false, int room = 0) {
    const int e = p.elem();
    int xch = 0;
    for (const Irrep& r : p.in1) xch += r.dim;
    const int xs = pad16((m.slice_full ? 32 * m.slice_cpl * xch : p.x_dim) * e);
    const int ws = p.unit ? 0 : pad16((m.slice_full ? 32 * (int)p.instr.size() : p.w_numel) * e);
    const int ep = m.slice_one ? 1 : 2;     // edges of a stage
    const int stage = 16 + (second ? 2 : 1) * (pad16(ep * p.y_dim * e) + ep * xs + ep * ws);     // (rows and cotangent rows)
    if (regs > 256) return false;
    m.slice_regs = regs;
    const int target = env_int("OEQ_B200_SLICE_WARPS_SM", std::max(regs, room) <= 124 ? 16 : (std::max(regs, room) <= 164 ? 12 : 8));
    m.slice_warps = m.n_slice * std::max(1, 4 / m.n_slice);
    if (m.slice_warps > 8) m.slice_warps = m.n_slice;
    for (int ctas = std::max(1, target / m.slice_warps); ctas >= 1; --ctas)
        for (int st = env_int("OEQ_B200_SLICE_STAGES", 3); st >= 2; --st) {
            const int smem = m.slice_warps * (st * stage + warp_bytes) + cta_bytes;
            if (smem <= SMEM_LIMIT && ctas * (smem + 1024) <= SMEM_LIMIT + 1024) {
                m.min_ctas = ctas;
                m.slice_stages = st;
                m.slice_smem = smem;
                return true;
            }
        }
    return false;
}

// Estimated registers up to which edge sums keep products per receiver, though that may leave fewer warps than the per-edge form:
// 800 k edges, per edge / sums, forward, 64x(0e+1o+2e) with 0e..3o (16 against 8 warps per SM) 681 / 534 us, FP64 with 0e+1o+2e
// (12 against 8) 878 / 705; backward, FP64 32x(0e+1o+2e) with 0e+1o 842 / 847, 128x(0e+1o) with 0e+1o+2e 1736 / 1422.
constexpr int OUTER_REGS = 240;

// Pairs of first- and second-input components of a channel, of the irreps that have a path: the measure of the register
// estimates.  (The pairs with a coefficient are what the kernels keep, but as a measure they give some kernels four warps per
// scheduler where three are faster: 64x(0e+1o) x (0e+1o+2e) -> 64x(0e+1o+2e), 800 k edges, backward 351 -> 376 us.)
int outer_pairs(const Problem& p) {
    std::set<std::pair<int, int>> seen;
    int n = 0;
    for (const Instr& i : p.instr)
        if (seen.insert({i.i1, i.i2}).second) n += p.in1[i.i1].dim * p.in2[i.i2].dim;
    return n;
}

// Pairs of components that have a coefficient: the products that the edge sums keep.
int coefficient_pairs(const Problem& p) {
    std::set<std::tuple<int, int, int, int>> seen;
    for (const Instr& t : p.instr)
        for (size_t n = 0; n < t.cv.size(); ++n) seen.insert(std::make_tuple(t.i1, t.i2, t.ci[n], t.cj[n]));
    return (int)seen.size();
}

// FP64 edge sums with few products per value of the row: an atomic backward pass is bound by its additions, 8 bytes each.  For
// x values per channel (128 channels, 200 k edges) it takes ~ 88 x us, the group kernel, which adds whole rows, ~ 130 + 32 x + 6.5
// per product.
bool bound_by_additions(const Problem& p) {
    int x = 0;
    for (const Irrep& r : p.in1) x += r.dim;
    return p.dtype == OEQ_F64 && coefficient_pairs(p) <= 9 * x - 20;
}

// The forward sums of products save the coefficient FMAs and the additions to the row, but take one edge at a time where the
// per-edge form of FP32 packs two: twice the reads of Y and about 20 operations per edge are lost.  800 k edges of 64 channels,
// per edge / sums of products: 64x(0e+1o+2e) to a scalar 220 / 261 us (12 operations saved), 0e+1o with 0e+1o 171 / 187 (18), with
// 0e+1o+2e to 0e+1o 206 / 228 (32, and 9 values of Y), 0e+1o+2e with 0e 226 / 240 (18); 0e+1o with 0e+1o to 0e+1o+2e 204 / 202 (34),
// 0e+1o+2e with 0e+1o+2e to 0e+1o 306 / 308 (52), with 0e+1o 314 / 292 (58).  FP64 has no packed form: 0e+1o 240 / 225.
bool outer_forward_pays(const Problem& p) {
    if (p.dtype == OEQ_F64) return true;
    int saved = 0;
    for (const Instr& t : p.instr) saved += (int)t.cv.size() + p.out[t.io].dim;
    return saved > 2 * p.y_dim + 20;
}

int build_slice_fwd(const Problem& p, bool deterministic, Kernel& k) {
    Mapping& m = k.map;
    if (!slice_shape(p, m)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not have the shape of the slice kernels");
    int zpc = 0, d1 = 1, tmax = 1, d3 = 1;
    for (const Irrep& r : p.out) { zpc += r.dim; d3 = std::max(d3, r.dim); }
    for (const Irrep& r : p.in1) d1 = std::max(d1, r.dim);
    for (size_t a = 0; a < p.in1.size(); ++a)
        for (size_t b = 0; b < p.in2.size(); ++b) {
            int t = 0;
            for (const Instr& i : p.instr)
                if (i.i1 == (int)a && i.i2 == (int)b) t += p.out[i.io].dim;
            tmax = std::max(tmax, t);
        }
    const int w = p.elem() / 4;
    int regs = zpc * w + 2 * (p.y_dim + d1 + tmax) + 24;
    const int outer = w * (outer_pairs(p) + p.y_dim + d1) + 28;
    m.slice_outer = p.unit && outer <= OUTER_REGS && outer_forward_pays(p);
    if (m.slice_outer) regs = outer;
    if (!slice_fit(p, m, regs, pad16(32 * d3 * p.elem()), 0)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not fit the slice kernels");
    m.mulg = 32;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    assign_partitions(p, false, m);
    int rc = compile_kernel(descriptor_text(p, m), "uvu_slice_kernels.cuh", deterministic ? K_SLICE_FWD_DET : K_SLICE_FWD_ATOMIC, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// Backward edge sums of rows of 64, 128 ... channels: two channels per lane share the walk, the second input and the sum of dY.
// 64x(0e+1o+2e), 400 k edges, forward and backward 1 028 -> 1 010 us; the forward pass alone gains 9 of 269 us there but loses
// 2 of 30 us on graphs of some hundred edges (fewer, longer walks) and keeps one channel.  One / two channels, 800 k edges: FP32
// 256x(0e+1o+2e) 3947 / 3085, 64x(0e+1o) 357 / 290; FP64 64x(0e+1o) with 0e+1o, deterministic, 935 / 753, 128x(0e+1o) with 0e+1o+2e,
// atomic, 1760 / 1422, 64x(0e+1o+2e) with 0e+1o, deterministic, 1707 / 1595.  Not where an atomic pass waits for its additions and
// would have fewer warps to wait with: the last one, atomic, 1607 / 1687; with 0e+1o+2e to 0e+1o, 200 k edges, 390 / 415.
bool two_channels_per_lane(Mapping& m, int regs) {
    if (!m.slice_full || m.n_slice % 2 || regs > OUTER_REGS) return false;
    m.slice_cpl = 2;
    m.n_slice /= 2;
    return true;
}

int build_slice_bwd(const Problem& p, bool deterministic, Kernel& k) {
    Mapping& m = k.map;
    if (!env_int("OEQ_B200_BWD_RECV", 1) || !slice_shape(p, m)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not have the shape of the slice kernels");
    int zpc = 0, d1 = 1, d2 = 1;
    for (const Irrep& r : p.out) zpc += r.dim;
    for (const Irrep& r : p.in1) d1 = std::max(d1, r.dim);
    for (const Irrep& r : p.in2) d2 = std::max(d2, r.dim);
    const int e = p.elem(), w = e / 4;      // registers of a value
    int per = 3 - w;                        // edges computed together
    int regs = w * (zpc + per * (2 * p.y_dim + 3 * d1 + d2)) + 12;
    const int outer = w * (outer_pairs(p) + per * (2 * p.y_dim + 2 * d1)) + 24;
    m.slice_outer = p.unit && outer <= OUTER_REGS;
    if (m.slice_outer) regs = outer;
    const int two = w * (2 * outer_pairs(p) + 2 * p.y_dim + 4 * d1) + 24;
    const bool waits = !deterministic && two > 164 && bound_by_additions(p);
    if (m.slice_outer && !waits && two_channels_per_lane(m, two)) {
        regs = two;
        per = 1;
    }
    int pitch = 8;
    while (pitch < 32 && pitch < per * p.y_dim) pitch *= 2;
    if (per * p.y_dim > 32) pitch = (per * p.y_dim + 31) / 32 * 32;
    const int groups = m.n_slice >= 4 ? 1 : 4 / m.n_slice;
    const int dyg = m.n_slice > 1 ? 2 * m.n_slice * pitch * e : 0;
    // FP64 rows with weights of their own take up to 1.6 times the estimate; with more warps they spill to an L1 that shared memory
    // leaves little of (16x(0e+1o+2e) with 0e+1o+2e: 108 bytes a thread).  200 k edges, atomic, 16 / 12 / 8 warps per SM (what
    // narrow rows have the shared memory for): 8x(0e+1o+2e) with 0e+1o+2e (estimate 158, 35 sums of the receiver)
    // 499 / 316 / 237 us, 8x(0e..3o) with 0e+1o (156, 40) 546 / 290 / 230, 8x(1o+2e) with 0e+1o+2e (136, 24) 280 / 210 / 179; with
    // 0e..3o to 8x(0e+1o) (156, 18) 359 / 196 / 208; 8x(0e+1o) with 0e+1o+2e to 8x(0e+1o+2e) (118, 21) 206 / 140 / 159, 8x(0e+2e)
    // with 0e+2e (110, 17) 177 / 138 / 157; 8x(0e+1o+2e) with 0e+1o (106, 21) 138 / 146 / 165.
    int room = 0;
    if (e == 8 && !p.unit) room = regs > 134 && zpc >= 24 ? 256 : (regs > 108 ? 126 : 0);
    if (!slice_fit(p, m, regs, 32 * pitch * e, groups * dyg, false, room)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not fit the slice kernels");
    m.mulg = 32;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    assign_partitions(p, true, m);
    int rc = compile_kernel(descriptor_text(p, m), "uvu_slice_kernels.cuh", deterministic ? K_SLICE_BWD_DET : K_SLICE_BWD_ATOMIC, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// Second derivatives of the convolution in slices: the gradient with respect to dZ (forward walk), or those with
// respect to X, Y, W (backward walk).
constexpr int K_SLICE_DBL_Z_DET = 54, K_SLICE_DBL_Z_ATOMIC = 55, K_SLICE_DBL_G_DET = 56, K_SLICE_DBL_G_ATOMIC = 57;

int build_slice_dbl(const Problem& p, bool deterministic, bool grads, Kernel& k) {
    Mapping& m = k.map;
    if (p.unit || !slice_shape(p, m)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not have the shape of the slice kernels");
    int zpc = 0, d1 = 1, d2 = 1, d3 = 1;
    for (const Irrep& r : p.out) { zpc += r.dim; d3 = std::max(d3, r.dim); }
    for (const Irrep& r : p.in1) d1 = std::max(d1, r.dim);
    for (const Irrep& r : p.in2) d2 = std::max(d2, r.dim);
    const int e = p.elem(), w = e / 4;
    // A stage of two edges and their cotangents, or of one: where two leave shared memory for fewer warps than the registers do
    // (FP64), or computing two together takes too many registers (FP32).  Forward and both derivatives, FP64, deterministic:
    // 128x(0e+1o+2e) x (0e..3o), 1 000 nodes / 28 k edges 1 304 -> 1 162 us; 32x(0e+1o+2e), 3 000 / 111 k 977 -> 894; FP32
    // 128x(0e..3o), group kernel before, 1 000 / 30 k 1 922 -> 1 419.  The two launches alone, FP32 128x(0e..3o), group / slices,
    // 30 k edges 1406 / 933, 990 k 36 405 / 28 975, atomic 36 913 / 27 106; 96 channels (six warps) 30 k 1122 / 900, 600 k 15 723 / 16 962.
    // Not where two edges have three warps per scheduler already (FP64 96x(0e+1o), 196 k edges, two / one edges 905 / 947), nor,
    // in the deterministic forward walk of rows of one slice, two: each warp takes a run there, and twice the warps leave more of
    // them with one receiver more than others (16x(0e+1o+2e), 28 k edges 138 / 178, 196 k 634 / 863; 20x(0e+1o+2e) x (0e+1o) 105 / 122).
    auto fit = [&](bool one) {
        const int per = one ? 1 : 3 - w;        // edges computed together
        m.slice_one = one;
        const int regs = w * (zpc + per * (grads ? 2 * p.y_dim + 6 * d1 + d2 : 2 * p.y_dim + 4 * d1 + 2)) + 12;
        int pitch = 8;
        while (pitch < 32 && pitch < per * p.y_dim) pitch *= 2;
        if (per * p.y_dim > 32) pitch = (per * p.y_dim + 31) / 32 * 32;
        const int groups = m.n_slice >= 4 ? 1 : 4 / m.n_slice;
        const int dyg = m.n_slice > 1 ? 2 * m.n_slice * pitch * e : 0;
        return slice_fit(p, m, regs, grads ? 32 * pitch * e : pad16(32 * d3 * e), grads ? groups * dyg : 0, true);
    };
    const bool pair = fit(false);
    if (!pair || w == 2) {
        const Mapping two = m;
        const bool one = fit(true);
        const int warps1 = m.min_ctas * m.slice_warps, warps2 = two.min_ctas * two.slice_warps;
        const bool keep = pair && warps2 >= (deterministic && !grads && m.n_slice == 1 ? 8 : 12);
        if (!pair && !one) return fail(OEQ_ERR_UNSUPPORTED, "problem does not fit the slice kernels");
        if (!one || (pair && (keep || warps1 <= warps2))) m = two;
    }
    m.mulg = 32;
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    assign_partitions(p, grads, m);
    const int kind = grads ? (deterministic ? K_SLICE_DBL_G_DET : K_SLICE_DBL_G_ATOMIC) : (deterministic ? K_SLICE_DBL_Z_DET : K_SLICE_DBL_Z_ATOMIC);
    int rc = compile_kernel(descriptor_text(p, m), "uvu_slice_kernels.cuh", kind, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// Where a thread of the backward slice kernel needs more than 200 registers (two warps per scheduler) for rows of several
// slices, the receiver-order group kernel with its staging warps is the faster one once the edges fill the machine.
// MACE-large, group / slice kernel in us: atomic 30 k edges 374 / 325, 65 k 601 / 636, 1.2 M 10211 / 11278; deterministic, with
// the row sum beside later launches on large lists only, 65 k 886 / 736, 131 k 1451 / 1434, 263 k 2751 / 2828, 1.2 M
// 11987 / 13138.  128x(0e+1o+2e) in FP64 is within 2 % from 15 k to 66 k edges and 131 k on 1154 / 1256 (atomic).  A row
// of one slice is the slice kernel's at every size: 32x(0e..3o), 65 k edges 202 / 173, 1.2 M 3552 / 2804.
// Edge sums of products (no weights) stay with the slice kernel whatever their registers: 128x(0e+1o+2e) with 0e+1o+2e, 200 k
// edges atomic 558 / 368, deterministic 792 / 541, 256 channels 992 / 773, 64x(0e..3o) 753 / 310, 128x(0e..3o) 1096 / 658.
// But FP64 rows of more than 64 channels that are bound by their additions: 128x(0e+1o+2e) with 0e+1o (32 products) 574 / 798,
// to 0e (4) 433 / 775, with 0e+1o+2e to 0e+1o (37)
// 638 / 781, 128x(0e+2e) with 0e+2e (34) 499 / 517, 256x(0e+1o) with 0e+1o (10) 628 / 738; on the other side 128x(0e+1o+2e) with
// 0e+1o+2e (71) 941 / 929, 256x(0e+1o) with 0e+1o+2e (21) 830 / 724, 256x0e (1) 387 / 270.
bool recv_beside_slice(const Problem& p, bool has_slice, const Kernel& slice, bool deterministic) {
    if (!has_slice) return true;
    const Mapping& m = slice.map;
    if (!m.slice_outer) return m.slice_regs > 200 && m.n_slice > 1;
    return !deterministic && m.n_slice * m.slice_cpl > 2 && bound_by_additions(p);
}
long long recv_min_edges(bool deterministic) { return env_int("OEQ_B200_RECV_MIN_EDGES", deterministic ? 196608 : 49152); }

// Wide FP64 rows in the forward pass: the slice kernel gathers every row once per slice of 32 channels, which
// costs once the rows no longer fit in L2.  128x(0e+1o+2e), group / slice kernel, atomic: 5 000 nodes (46 MB) 695 / 636 us,
// 10 000 (92 MB) 1252 / 1277, 20 000 2422 / 2730; deterministic 659 / 592, 1159 / 1171, 2330 / 2422.
// (Edge sums of products read rows once per 32 channels too, but compute less: 128x(0e+1o+2e), 20 000 nodes, 2508 / 1373.)
bool group_forward_beside_slice(const Problem& p, const Kernel& slice) {
    return p.dtype == OEQ_F64 && !slice.map.slice_outer && slice.map.slice_regs > 160 && slice.map.n_slice > 2;
}
constexpr size_t GROUP_FORWARD_BYTES = 64u << 20;

// Problems for which fused second derivatives may exist (whether they fit is known once they are built).
bool conv_second_possible(const Problem& p) {
    Mapping m;
    return !p.unit && env_int("OEQ_B200_FUSED_DOUBLE_BACKWARD", 1) != 0 && (conv_double_backward_supported(p) || slice_shape(p, m));
}

// Both second-derivative kernels of a convolution: slice kernels, or the group kernels where a row does not fit them.
int build_conv_dbl(const Problem& p, bool deterministic, Kernel& z, Kernel& g) {
    int rc = build_slice_dbl(p, deterministic, false, z);
    if (!rc) rc = build_slice_dbl(p, deterministic, true, g);
    if (rc != OEQ_ERR_UNSUPPORTED) return rc;
    z = Kernel();
    g = Kernel();
    if (!conv_double_backward_supported(p)) return rc;
    rc = build_uvu_dblc(p, deterministic, false, z);
    return rc ? rc : build_uvu_dblc(p, deterministic, true, g);
}

constexpr int K_FWD_DET_TC = 30, K_FWD_ATOMIC_TC = 31;

int build_uvu_tc(const Problem& p, bool deterministic, Kernel& k) {
    if (!uvu_tc_geometry(p, k.tc_geo)) return fail(OEQ_ERR_UNSUPPORTED, "problem does not qualify for the tensor-core forward pass");
    Mapping& m = k.map;
    m.mulg = 128; m.nch = 1; m.ng = 1; m.producer = 1; m.min_ctas = 1;
    m.ps = std::max(1, std::min({2, (int)p.out.size(), env_int("OEQ_B200_TC_PARTS", 2)}));
    m.z_ph_begin = {0, p.z_dim};
    m.w_ph_begin = {0, p.w_numel};
    m.phase_of_instr.assign(p.instr.size(), 0);
    m.tc_tables = true;
    assign_partitions(p, false, m);
    const UvuTcColumns cols = uvu_tc_columns(p, m.part_of_out, m.ps);
    if (!uvu_tc_geometry(p, k.tc_geo, cols.part_col.back()))
        return fail(OEQ_ERR_UNSUPPORTED, "problem does not fit the tensor-core forward pass");
    k.is_uvu_tc = true;
    int rc = compile_kernel(descriptor_text(p, m), "uvu_tc_kernels.cuh", deterministic ? K_FWD_DET_TC : K_FWD_ATOMIC_TC, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

constexpr int K_UVW_FWD = 10, K_UVW_BWD = 11;

int build_uvw(const Problem& p, int kind, Kernel& k) {
    k.is_uvw = true;
    int rc = choose_uvw(p, kind == K_UVW_BWD, k.uvw);
    if (rc) return rc;
    // the uvu mapping tables are emitted with neutral values so that one descriptor format serves both
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    rc = compile_kernel(descriptor_text(p, k.map, &k.uvw), "uvw_kernels.cuh", kind, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// ---- tensor-core forward for 'uvw' (mirrors the constexpr geometry of uvw_tc_kernels.cuh)
constexpr int K_UVW_TC_FWD = 20;

struct TcGeometry {
    size_t packed_bytes = 0;
    int smem = 0;
    unsigned outputs = 1;
    unsigned paths = 1;                     // instructions (the weights of each are packed by blocks of their own)
    int producers = 16, epilogues = 1;      // producer warps, groups of four epilogue warps
    int dealt_rows_per_sm = 200;            // batches whose chunks are dealt over the CTAs (launch_uvw_tc)
    int threads() const { return 32 * (producers + 1 + 4 * epilogues); }
};

// `pad`: output multiplicities may be rounded up to 16 (the products W dZ of the backward pass).
bool uvw_tc_geometry(const Problem& p, TcGeometry& g, bool pad = false) {
    if (p.mode != OEQ_MODE_UVW || !p.shared || p.dtype != OEQ_F32) return false;
    if (!env_int("OEQ_B200_UVW_TC", 1)) return false;
    int w_max = 0, mw_max = 16;
    size_t total = 0;
    for (size_t o = 0; o < p.out.size(); ++o) {
        int blocks = 0;
        for (const Instr& t : p.instr)
            if (t.io == (int)o) {
                if (p.in2[t.i2].mul != 1) return false;
                blocks += (p.in1[t.i1].mul + 31) / 32;
            }
        if (blocks == 0) continue;
        const int mw = (p.out[o].mul + 15) / 16 * 16;
        if ((!pad && mw != p.out[o].mul) || mw > 256 || p.out[o].dim > 64) return false;
        const int bytes = blocks * 2 * mw * 128;
        w_max = std::max(w_max, bytes);
        mw_max = std::max(mw_max, mw);
        total += bytes;
    }
    if (total == 0) return false;
    for (const Irrep& r : p.in1)
        if (r.mul > 32) g.dealt_rows_per_sm = 160;
    g.producers = p.unit_y ? 8 : 16;
    g.epilogues = p.unit_y ? 2 : 1;
    const int off_w = 2 * 2 * 128 * 128;
    const int off_stg = off_w + (w_max + 1023) / 1024 * 1024;
    const int pitch = (g.epilogues > 1 ? 32 : std::min(mw_max, 64)) + 1;
    const int off_bar = off_stg + g.epilogues * ((128 * pitch * 4 + 15) / 16 * 16);
    g.smem = off_bar + (2 * 2 + 2 * 32 + 2) * 8 + 16 + 1024;
    g.packed_bytes = total;
    g.paths = (unsigned)p.instr.size();
    g.outputs = (unsigned)p.out.size();
    return g.smem <= SMEM_LIMIT;
}

int build_uvw_tc(const Problem& p, const TcGeometry& g, Kernel& k) {
    k.is_uvw = true;
    int rc = choose_uvw(p, false, k.uvw);
    if (rc) return rc;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    const std::string roles = "#define TC_PW " + std::to_string(g.producers) + "\n#define TC_EPI " + std::to_string(g.epilogues) + "\n";
    rc = compile_kernel(descriptor_text(p, k.map, &k.uvw) + roles, "uvw_tc_kernels.cuh", K_UVW_TC_FWD, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// ---- the same with the weights in tensor memory (mirrors the constexpr geometry of uvw_ts_kernels.cuh): at most 64 output
// channels per irrep, 256 input channels over the paths into one, rows of X in whole 16-byte pieces of four channels.
constexpr int K_UVW_TS_FWD = 22, TS_ROWS = 16, TS_STAGES = 4, TS_THREADS = 21 * 32;

bool uvw_ts_geometry(const Problem& p, int& smem) {
    TcGeometry g;
    if (p.unit_y || p.transposed_w || !uvw_tc_geometry(p, g) || p.x_dim % 4) return false;
    int data = 0;
    for (size_t o = 0; o < p.out.size(); ++o) {
        int slices = 0;
        for (const Instr& t : p.instr)
            if (t.io == (int)o) slices += (p.in1[t.i1].mul + 31) / 32;
        if (slices == 0) continue;
        if (p.out[o].mul > 64 || p.out[o].dim > 8 || slices > 8) return false;
        data = std::max(data, TS_ROWS * p.out[o].dim * (4 * 2 * 128 + 2 * p.out[o].mul * 4));      // stages, rows of Z
    }
    for (const Irrep& r : p.in1)
        if (r.mul % 4 || r.off % 4) return false;
    smem = data + 2 * TS_ROWS * (p.x_dim + p.y_dim) * 4 + (int)p.out.size() * (2 * 4 + 2 * 4 + 2 * 4) * 8 + 16 + 1024;
    return smem <= SMEM_LIMIT;
}

// Whether that kernel is the faster one, by the work of the problem and not of the batch: a row has the same bits in every batch.
// Time of either, in units of 10 ns per 100 000 rows (fitted to 42 problems, all within 25 %): this kernel's drain costs a tile of 16 rows the same for
// one slice of 32 input channels as for eight; the other kernel's producers read rows of X with a stride of 2 l + 1 values, slice by
// slice, and its drain goes with the values of Z.
// Measured, us for 100 000 rows, shared / tensor memory (at 1 000 rows; estimates tensor / shared):
//   with 0e+1o+2e: 64x(0e+1o+2e) 413 / 272 (30 / 23; 0.72), 16x 194 / 183 (1.06), 48x(0e+1o+2e) to 64x0e 120 / 66 (0.68)
//   with 0e+1o: 64x(0e+1o+2e) 237 / 209 (0.84), 64x(0e+1o) 106 / 109 (15.3 / 10.6; 1.07), 16x 52 / 90 (13.3 / 10.2; 1.95)
//   with 0e: 256x1o to 64x1o 124 / 94 (0.72), 96x 64.5 / 63.5 (0.98), 64x 56.3 / 57.3 (15.3 / 10.2; 1.13); 256x0e to 64x0e 61 / 61 (17.5 /
//     12.3; 1.16), 128x0e 36 / 49 (15.3 / 10.2; 1.55), 32x0e to 32x0e 19.4 / 37.5 (13.3 / 10.2; 3.8); 64x(0e+1o+2e) 136 / 171 (1.13)
// Up to 1.1 this kernel loses at most 3 % at 100 000 rows, none up to 30 000, and is 4 to 47 % faster up to 4 000.
bool uvw_ts_faster(const Problem& p) {
    long long tensor = 0, shared = 0;
    std::vector<bool> used(p.out.size());
    for (const Instr& t : p.instr) {
        const long long slices = (p.in1[t.i1].mul + 31) / 32, d1 = p.in1[t.i1].dim, d3 = p.out[t.io].dim, n = (long long)t.cv.size();
        tensor += slices * (170 + 78 * d3 + 47 * d1 + 30 * n);
        shared += slices * (112 + 341 * d1 + 44 * n);
        used[t.io] = true;
    }
    for (size_t o = 0; o < p.out.size(); ++o)
        if (used[o]) {
            tensor += 2240 + 420 * p.out[o].dim;
            shared += 9 * p.out[o].dim * p.out[o].mul;
        }
    return 10 * tensor <= 11 * shared;
}

int build_uvw_ts(const Problem& p, Kernel& k) {
    k.is_uvw = true;
    int rc = choose_uvw(p, false, k.uvw);
    if (rc) return rc;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    rc = compile_kernel(descriptor_text(p, k.map, &k.uvw), "uvw_ts_kernels.cuh", K_UVW_TS_FWD, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// ---- weight gradient from rows formed a batch row per lane (mirrors uvw_ts_dw_kernels.cuh)
constexpr int K_UVW_TS_DW = 23, TG_ROWS = 8;

bool uvw_ts_dw_geometry(const Problem& p, int& smem) {
    int fwd = 0;
    if (!uvw_ts_geometry(p, fwd) || p.z_dim % 4 || !env_int("OEQ_B200_UVW_TC_BWD", 1)) return false;
    int data = 0;
    for (size_t o = 0; o < p.out.size(); ++o) {
        bool paths = false;
        for (const Instr& t : p.instr) paths |= t.io == (int)o;
        if (!paths) continue;
        if (p.out[o].off % 4) return false;
        data = std::max(data, 1024 * p.out[o].dim * (2 * 8 + 2 * ((2 * p.out[o].mul + 31) / 32)) +      // slots of T, of dZ, inputs
                                  2 * TG_ROWS * (p.x_dim + p.y_dim + p.out[o].mul * p.out[o].dim) * 4);
    }
    // (`smem` is that of the wider kernel until this one is taken)
    const int bytes = std::max(data, 222 * 1024) + (int)p.out.size() * (2 * 2 + 2 * 2 + 2 * 4 + 2 * 3) * 8 + 16 + 1024;
    if (bytes > SMEM_LIMIT) return false;
    smem = bytes;
    return true;
}

int build_uvw_ts_dw(const Problem& p, Kernel& k) {
    k.is_uvw = true;
    int rc = choose_uvw(p, true, k.uvw);
    if (rc) return rc;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    rc = compile_kernel(descriptor_text(p, k.map, &k.uvw), "uvw_ts_dw_kernels.cuh", K_UVW_TS_DW, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// ---- tensor-core backward for 'uvw': the weight gradient (mirrors the constexpr geometry of uvw_tc_bwd_kernels.cuh)
constexpr int K_UVW_TC_DW = 21;

bool uvw_tc_dw_geometry(const Problem& p, int& smem, int& threads) {
    TcGeometry fwd;
    if (!uvw_tc_geometry(p, fwd)) return false;          // same class of problems as the forward pass
    if (!env_int("OEQ_B200_UVW_TC_BWD", 1)) return false;
    int mw_max = 16;
    for (const Irrep& r : p.out) {
        mw_max = std::max(mw_max, r.mul);
        if (r.dim > 32) return false;                    // a stage holds at least one batch row
    }
    for (const Instr& t : p.instr)
        if (p.in1[t.i1].mul > 128) return false;
    if (mw_max > 128) return false;
    const int stage = 2 * 128 * 128 + 2 * mw_max * 128;
    const int stages = std::min(4, (200 * 1024) / stage);
    if (stages < 2) return false;
    smem = stages * stage + (2 * stages + 4) * 8 + 16 + 1024;
    threads = 32 * (4 * stages + 1 + 4);                 // four producer warps per stage, MMA issuer, epilogue
    return smem <= SMEM_LIMIT;
}

// Which of the two weight-gradient kernels a batch takes.  The wider one (uvw_tc_bwd_kernels.cuh) has an MMA tile of 128 rows for a group
// of two paths (one where they have more than 64 channels), a stage of 32 (row, component) pairs for each, and deals the groups over the
// CTAs while those suffice; the other one (uvw_ts_dw_kernels.cuh) sums four slices of 32 channels per MMA, eight batch rows at a time.
//   Few rows: tiles of eight rows times the outputs are few CTAs, each with all slices of its output, against groups that are dealt.
//     wider / other in us, with the sum over CTAs: 64x(0e+1o+2e) with 0e+1o+2e (22 slices) 20 rows 19.9 / 31.7, 500 23.7 / 37.9, but 1 000
//     (groups no longer dealt) 64.5 / 40; with 0e+1o (14 slices) 20 rows 19.5 / 25.6, 1 000 25.3 / 31.7, 2 000 50 / 34; 32x(0e+1o+2e)
//     with 0e+1o+2e (11) 20 rows 17.4 / 23.5; 64x(0e+1o) with 0e+1o (8 slices, two outputs) 200 rows 21.5 / 21.5; but 16x(0e+1o) (4)
//     17.2 / 13.3, 16x(0e+1o+2e+3o) with 0e (4 slices, four outputs) 23.6 / 19.5
//   Many rows: a scalar output has one MMA of K = 8 per tile and slices, and the other kernel does its rounds for that; outputs of more
//     components gain.  100 000 rows, with 0e: 64x0e to 16x0e 58 / 73, 128x0e to 64x0e 69 / 84, 32x0e 60 / 65, 128x1o to 64x1o 99 / 107, but
//     64x1o 118 / 86, 32x2e 173 / 81, 32x3o 245 / 90; 64x(0e+1o) with 0e+1o 159 / 176, 16x 158 / 151; at 10 000 rows 21.5 / 19.5, 27.6 / 26.7,
//     21.5 / 19.5, 29.7 / 29.2, ..., 42 / 38.  The sum over the outputs below is the loss at 100 000 rows in us, roughly.
struct DwChoice {
    unsigned groups = 0;                    // of paths, in the wider kernel
    bool few = false, many = false;         // the wider kernel is the faster one at few, at many rows
    long long wider_ctas(long long batch, int sms) const { return std::max<long long>(1, std::min<long long>(sms, (batch + 31) / 32)); }
    bool wider(long long batch, int sms) const {
        return (few && wider_ctas(batch, sms) * groups <= sms) || (many && batch > 100ll * sms);
    }
};

DwChoice uvw_dw_choice(const Problem& p) {
    DwChoice c;
    int slices_all = 0, outputs = 0, loss = 0;
    for (size_t o = 0; o < p.out.size(); ++o) {
        unsigned paths = 0, per = 2;
        int slices = 0;
        for (const Instr& t : p.instr)
            if (t.io == (int)o) {
                ++paths;
                slices += (p.in1[t.i1].mul + 31) / 32;
                if (p.in1[t.i1].mul > 64) per = 1;
            }
        if (!paths) continue;
        const unsigned groups = (paths + per - 1) / per;
        const int dim = p.out[o].dim;
        c.groups += groups;
        slices_all += slices;
        ++outputs;
        if (groups > 1) loss -= dim == 1 ? 30 : 60;
        else if (dim == 1) loss += 12;
        else if (slices == 4) loss += dim == 3 ? 7 : -5;
        else loss -= dim == 3 ? 25 : 60;
    }
    c.few = c.groups > 1 && slices_all > 3 * outputs;
    c.many = loss > 0;
    return c;
}

// ---- dX and dY of the same class of problems in two steps over a scratch array dT [row][path][u][k]:
//   dT_p[b,u,k] = sum_w W_p[u,w] dZ[b,w,k]: a 'uvw' forward pass from the output irreps, with the second input the
//   number 1 and the weights transposed, one output block per path (`product`);
//   dX, dY from dT: the channel-wise backward pass with every weight 1 (`channels`).
void uvw_gradient_problems(const Problem& p, Problem& product, Problem& channels) {
    product = Problem();
    product.mode = OEQ_MODE_UVW;
    product.shared = 1;
    product.unit_y = product.transposed_w = true;
    product.in1 = p.out;
    product.x_dim = p.z_dim;
    product.in2 = {Irrep{1, 0, 1, 1, 0}};
    product.y_dim = 1;
    product.w_numel = p.w_numel;
    channels = p;
    channels.mode = OEQ_MODE_UVU;
    channels.shared = 0;
    channels.unit = 1;
    channels.out.assign(p.instr.size(), Irrep());
    int off = 0;
    for (size_t o = 0; o < p.out.size(); ++o) {
        // the paths into o read the same dZ tiles: joined in one output block of up to 256 channels, as far as the
        // weights of a block fit 128 KB of shared memory
        const int slices = (p.out[o].mul + 31) / 32, cap = std::min(256, 131072 / (slices * 256) / 16 * 16);
        bool open = false;
        for (size_t n = 0; n < p.instr.size(); ++n) {
            const Instr& t = p.instr[n];
            if (t.io != (int)o) continue;
            const int mul = p.in1[t.i1].mul, dim = p.out[o].dim;
            if (!open || product.out.back().mul + mul > cap) {
                Irrep block = p.out[o];
                block.mul = 0;
                block.off = off;
                product.out.push_back(block);
                Instr q = t;
                q.i1 = (int)o; q.i2 = 0; q.io = (int)product.out.size() - 1; q.pw = 1.0;
                q.ci.clear(); q.cj.clear(); q.ck.clear(); q.cv.clear();
                for (int k = 0; k < dim; ++k) { q.ci.push_back(k); q.cj.push_back(0); q.ck.push_back(k); q.cv.push_back(1.0); }
                product.instr.push_back(q);
                product.subs.emplace_back();
                open = true;
            }
            Irrep& block = product.out.back();
            product.subs.back().push_back({block.mul, mul, t.w_off});
            channels.out[n] = p.out[o];
            channels.out[n].mul = mul;
            channels.out[n].off = off;
            channels.instr[n].io = (int)n;
            channels.instr[n].mode = OEQ_MODE_UVU;
            block.mul += mul;
            off += mul * dim;
        }
    }
    product.z_dim = channels.z_dim = off;
}
// Scratch rows: all of them up to 1 GiB, then blocks.
constexpr size_t UVW_DT_BYTES = 1u << 30;

int build_uvw_tc_bwd(const Problem& p, int kernel_id, Kernel& k) {
    k.is_uvw = true;
    int rc = choose_uvw(p, true, k.uvw);
    if (rc) return rc;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    rc = compile_kernel(descriptor_text(p, k.map, &k.uvw), "uvw_tc_bwd_kernels.cuh", kernel_id, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// One row per CTA for 'uvw' with per-row weights (uvw_row_kernels.cuh): T of a row (and dT) in shared memory, eight
// input channels of a path in registers.  Rows that take more keep the tiled kernel.
constexpr int K_UVW_ROW_FWD = 12, K_UVW_ROW_BWD = 13, UVW_ROW_WARPS = 8;

int uvw_row_smem(const Problem& p, bool bwd) {
    auto r4 = [](long long n) { return (n + 3) / 4 * 4; };
    long long t = 0;
    for (const Instr& i : p.instr) t += (long long)p.in1[i.i1].mul * p.in2[i.i2].mul * p.out[i.io].dim;
    const long long e = r4(p.x_dim) + r4(p.y_dim) + r4(p.z_dim) + r4(t) * (bwd ? 2 : 1) + (bwd ? UVW_ROW_WARPS * p.y_dim : 0);
    return (int)std::min<long long>(e * p.elem(), 1ll << 30);
}

bool uvw_row_supported(const Problem& p) {
    if (p.mode != OEQ_MODE_UVW || p.shared) return false;
    for (const Irrep& r : p.out)
        if (r.dim * 8 * (p.elem() / 4) > 128) return false;
    return uvw_row_smem(p, true) <= 100 * 1024;
}

// Rows per SM up to which the row kernel is the faster one (0: always).  It pays a CTA's barriers and phases per row, the
// tiled kernel shares them among 16 rows; with few weights a row that is what counts once every SM has rows enough.
// Measured, tiled against row kernel in us (30 000 rows unless stated, second input 0e+1o..., rows that are not staged):
//   forward: FP32 by the input channels of all paths: 8x(0e+1o) (32) 51 / 84, 12x(0e+1o) (48) 121 / 141, 8 -> 64 channels (32)
//     74 / 102, but 16x(0e+1o) (64) 225 / 127, 4x(0e..3o) (136) 199 / 174; 2 000 rows 12 / 12 and 14 / 16.  FP64, whose tiled
//     kernel is slower: 1x(0e+1o) (4) 20 / 45, but 4x(0e+1o) (16) 74 / 66; one tile of output channels keeps one warp of eight
//     busy: 128x0e -> 4x0e 317 / 504.
//   backward: by the weights per path: FP32 4x(0e+1o) (16) 53 / 123, 4x(0e..3o) (16) 657 / 1000, 8x(0e+1o+2e) (64) 260 / 299,
//     but 12x(0e+1o) (144) 215 / 131; FP64 4x(0e..3o) 961 / 3029 (1 000 rows 92 / 123), 8x(0e+1o+2e) (64) 668 / 897 (2 000 rows
//     57 / 70, 1 000 rows 55 / 41), but without l = 2 8x(0e+1o) (64) 221 / 154; fewer than eight output channels leave most lanes idle: 128x0e -> 4x0e 88 / 113.
// Staged rows (below) are faster than that, and the lines stand where they stood: 30 000 rows forward FP32 8x(0e+1o) 50 / 35, 12x 118 / 41,
//   4x 34 / 35, FP64 128x0e with 4x0e -> 4x0e 809 / 97; backward FP32 8x 92 / 72, the latter 346 / 158, but 4x 51 / 73; FP64 4x(0e..3o) 953 / 1061.
int uvw_row_limit(const Problem& p, bool bwd) {
    long long uv = 0, tiles = 0;
    int dim = 1, width = 0;
    for (const Instr& t : p.instr) uv += (long long)p.in1[t.i1].mul * p.in2[t.i2].mul;
    for (const Irrep& r : p.out) {
        tiles += (r.mul + 31) / 32;
        dim = std::max(dim, r.dim);
        width = std::max(width, r.mul);
    }
    const bool f64 = p.dtype == OEQ_F64;
    if (!bwd) return (f64 ? uv < 8 || tiles == 1 : uv < 64) ? 24 : 0;
    const long long per_path = p.w_numel / (long long)p.instr.size();
    if (per_path >= (f64 && dim <= 3 ? 48 : 144) && width >= 8) return 0;
    if (f64 && dim >= 5) return per_path < 32 ? 5 : 8;
    return per_path < 32 ? 8 : 64;
}

// Staged rows (uvw_row_kernels.cuh): bulk copies want rows of whole 16-byte pieces, and two stages have to leave room for a
// second CTA on an SM.  Shared memory of a CTA, 0 where a row does not qualify.
// Loads where a weight is used / staged, us, 2 011 rows: forward 4x(0e+1o) with 0e+1o 6.5 / 6.4, 32x 24 / 10, 16x(0e+1o) with 4x(0e+1o) 70 / 12, FP64 32x 39 / 15;
// backward 4x 8.4 / 8.4, 32x 18.8 / 16.7, 8x(0e..3o) with 0e..3o 87 / 47, FP64 16x 21 / 13, 32x0e with 4x0e 23 / 21.  30 shapes at 20 to 30 000 rows:
// none slower by more than a microsecond or 2 % (FP64 32x0e with 4x0e, backward, 30 000 rows 325 / 331).
constexpr int K_UVW_STAGED_FWD = 14, K_UVW_STAGED_BWD = 15, UVW_STAGED_BYTES = (228 * 1024) / 2 - 1024;
constexpr int UVW_STAGED_UNITS = 256;      // (the compiler deals them)

int uvw_staged_smem(const Problem& p, bool bwd) {
    const long long e = p.elem();
    for (long long n : {p.x_dim, p.y_dim, p.z_dim, p.w_numel})
        if (n * e % 16) return 0;
    auto r4 = [](long long n) { return (n + 3) / 4 * 4; };
    long long t = 0, parts = 0, units = 0;
    for (const Instr& i : p.instr) {
        const int mu = p.in1[i.i1].mul, mv = p.in2[i.i2].mul, mw = p.out[i.io].mul, d3 = p.out[i.io].dim;
        t += (long long)mu * mv * d3;
        for (int wc = 0; wc < mw; wc += 32) {
            const int wlen = std::min(32, mw - wc);
            parts += (long long)((mu + 31) / 32) * (32 / wlen) * wlen * d3;
        }
        units += bwd ? (long long)((mu + 15) / 16) * mv : (long long)((mu + 31) / 32) * ((mw + 31) / 32);
    }
    if (units > UVW_STAGED_UNITS) return 0;
    const long long stage = (long long)p.w_numel + p.x_dim + p.y_dim + (bwd ? p.z_dim : 0);
    const long long bytes = (2 * stage + r4(t) + r4(bwd ? r4(t) + 2 * UVW_ROW_WARPS * p.y_dim : parts)) * e + (bwd ? units * 48 : 0) + 16;
    return bytes <= UVW_STAGED_BYTES ? (int)bytes : 0;
}

int build_uvw_row(const Problem& p, bool bwd, Kernel& k) {
    const int staged = uvw_staged_smem(p, bwd);
    k.row_smem = staged ? staged : uvw_row_smem(p, bwd);
    k.is_uvw = k.is_uvw_row = true;
    k.uvw.tile_r = 1;       // (the tiled kernel's bodies are not compiled)
    k.uvw.threads = 32 * UVW_ROW_WARPS;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    const std::string rows = "namespace oeqd { constexpr int ROW_WARPS = " + std::to_string(UVW_ROW_WARPS) + "; }\n";
    int rc = compile_kernel(descriptor_text(p, k.map, &k.uvw) + rows, "uvw_row_kernels.cuh",
                            staged ? (bwd ? K_UVW_STAGED_BWD : K_UVW_STAGED_FWD) : (bwd ? K_UVW_ROW_BWD : K_UVW_ROW_FWD), k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// Both kernels of the two-step dX / dY (OEQ_ERR_UNSUPPORTED where a row does not fit them).
int build_uvw_gradients(const Problem& p, Problem& product, Problem& channels, TcGeometry& g, Kernel& kp, Kernel& kc) {
    uvw_gradient_problems(p, product, channels);
    if (!uvw_tc_geometry(product, g, true)) return fail(OEQ_ERR_UNSUPPORTED, "rows do not fit the tensor-core product");
    int rc = build_uvw_tc(product, g, kp);
    if (!rc) rc = build_uvu(channels, K_BWD_BATCH, kc);
    return rc;
}

// ---- FP64 with shared weights as register-tiled GEMMs (uvw_gemm_kernels.cuh).  Multiplicities below 16 would fill less
// than a quarter of a tile's edge and keep the tiled kernel.
constexpr int K_UVW_GEMM = 14, K_UVW_GEMM_DW = 15, GEMM_TILE = 64, GEMM_SMEM = 4 * 32 * 66 * 8;

bool uvw_gemm_supported(const Problem& p) {
    if (p.mode != OEQ_MODE_UVW || !p.shared || p.dtype != OEQ_F64) return false;
    for (const Irrep& r : p.in2)
        if (r.mul != 1) return false;
    for (const std::vector<Irrep>* v : {&p.in1, &p.out})
        for (const Irrep& r : *v)
            if (r.mul < 16 || r.dim > 32) return false;
    return true;
}

// Batches that the tiled kernel computes faster than the GEMMs, whose chain of chunks of 32 channels, each with a barrier,
// and whose three launches backward show where there is little to do.  Measured, tiled / GEMM in us:
//   forward, up to one wave of 16-row tiles (2 368 rows) and 4 096 products a row (8 192 with one path): 300 rows of 32x0e
//     8 / 12, 128x0e -> 64x0e 12 / 25, 16x(0e+1o) 12 / 14, but one row of 64 -> 16x(0e+1o) (8 192, four paths) 26 / 20; above
//     either line 128x0e -> 64x0e 5 000 rows 27 / 22, 16x(0e+1o+2e) (8 960) 27 / 18.
//     Half-filled tiles with l = 2 lose at many rows: 20x(0e+1o+2e), 60 000 rows 428 / 504, 25 000 rows 188 / 199, 20 000
//     158 / 160; 16 and 24 channels, 25 000 rows 180 / 174 and 233 / 221; 28x(0e+1o+2e) 617 / 606.  16x0e alone never fills a tile: 60 000 rows 29 / 33.
//   backward, from the 128 rows on that take two shares of the rows (and their sum): 300 rows of 16x(0e+1o) (2 048) 36 / 46,
//     32x0e 22 / 32; 64x0e (4 096) 46 / 38, one row of 16x(0e+1o) 32 / 17.
constexpr int GEMM_SMALL_FWD = 4096, GEMM_SMALL_FWD_ONE_PATH = 8192, GEMM_SMALL_BWD = 2048, GEMM_SMALL_ROWS_PER_SM = 16;

long long uvw_row_products(const Problem& p) {
    long long n = 0;
    for (const Instr& t : p.instr) n += (long long)p.in1[t.i1].mul * p.in2[t.i2].mul * p.out[t.io].mul * p.out[t.io].dim;
    return n;
}
// Rows per SM from which multiplicities below 28 with l >= 2 are for the tiled kernel (0: not one of them).
int gemm_narrow_rows_per_sm(const Problem& p) {
    int mul = 0, dim = 0;
    for (const std::vector<Irrep>* v : {&p.in1, &p.out})
        for (const Irrep& r : *v) mul = std::max(mul, r.mul);
    for (const Irrep& r : p.out) dim = std::max(dim, r.dim);
    return mul < 28 && dim >= 5 ? 200 : 0;
}
bool gemm_small_forward(const Problem& p) { return uvw_row_products(p) <= (p.instr.size() == 1 ? GEMM_SMALL_FWD_ONE_PATH : GEMM_SMALL_FWD); }
bool gemm_forward_tiled(const Problem& p, long long batch, long long sms) {
    if (uvw_row_products(p) <= 256 || (gemm_small_forward(p) && batch <= GEMM_SMALL_ROWS_PER_SM * sms)) return true;
    return gemm_narrow_rows_per_sm(p) && batch > gemm_narrow_rows_per_sm(p) * sms;
}
bool gemm_backward_tiled(const Problem& p, long long batch, long long sms) {
    return uvw_row_products(p) <= GEMM_SMALL_BWD && batch >= 128 && batch <= GEMM_SMALL_ROWS_PER_SM * sms;
}
// Whether any batch takes the tiled forward kernel (the backward one is there anyway, for small workspaces).
bool gemm_keeps_tiled(const Problem& p) { return gemm_small_forward(p) || gemm_narrow_rows_per_sm(p) > 0; }

int build_uvw_gemm(const Problem& p, int kernel_id, Kernel& k) {
    k.is_uvw = true;
    k.map.part_of_out.assign(p.out.size(), 0);
    k.map.part_of_instr.assign(p.instr.size(), 0);
    k.map.zr_off.assign(p.out.size(), 0);
    k.map.xr_off.assign(p.in1.size(), 0);
    k.uvw.threads = 256;
    int rc = compile_kernel(descriptor_text(p, k.map), "uvw_gemm_kernels.cuh", kernel_id, k.code);
    if (rc) return rc;
    k.compiled = true;
    return OEQ_OK;
}

// The three kernels of the backward pass: weight gradient, dT = W dZ, and dX, dY from dT.
int build_uvw_gemm_backward(const Problem& p, Problem& product, Problem& channels, Kernel& dw, Kernel& kp, Kernel& kc) {
    uvw_gradient_problems(p, product, channels);
    product.dtype = p.dtype;
    int rc = build_uvu(channels, K_BWD_BATCH, kc);
    if (!rc) rc = build_uvw_gemm(p, K_UVW_GEMM_DW, dw);
    if (!rc) rc = build_uvw_gemm(product, K_UVW_GEMM, kp);
    return rc;
}

// Shares of the rows in the weight gradient: about six CTAs per SM, 64 rows or more each.
long long gemm_shares(const Problem& p, long long batch, long long sm_count) {
    long long tiles = 0;
    for (const Instr& t : p.instr)
        tiles += (long long)((p.in1[t.i1].mul + GEMM_TILE - 1) / GEMM_TILE) * ((p.out[t.io].mul + GEMM_TILE - 1) / GEMM_TILE);
    return std::max<long long>(1, std::min((6 * sm_count + tiles - 1) / std::max<long long>(1, tiles), batch / 64));
}

// `row`: kernel with one row per CTA, where the problem has one; the kernel for the other batches is then optional.
int build_tp(const Problem& p, bool bwd, Kernel& k, Kernel& row) {
    if (uvw_row_supported(p)) {
        const int rc = build_uvw_row(p, bwd, row);
        if (rc || uvw_row_limit(p, bwd) == 0) return rc;
        const int tiled = build_uvw(p, bwd ? K_UVW_BWD : K_UVW_FWD, k);
        return tiled == OEQ_ERR_UNSUPPORTED ? OEQ_OK : tiled;
    }
    if (p.mode == OEQ_MODE_UVW) return build_uvw(p, bwd ? K_UVW_BWD : K_UVW_FWD, k);
    return build_uvu(p, bwd ? K_BWD_BATCH : K_FWD_BATCH, k);
}

int load_uvw(Kernel& k, const Problem& p, bool bwd) {
    if (k.loaded) return OEQ_OK;
    OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, k.is_uvw_row ? "oeq_uvw_row_kernel" : "oeq_uvw_kernel"));
    if (!k.is_uvw_row) OEQ_CUDA(cudaLibraryGetKernel(&k.reduce_fn, k.lib, "oeq_reduce_partials"));
    int dev = 0;
    OEQ_CUDA(cudaGetDevice(&dev));
    OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
    k.smem = k.is_uvw_row ? k.row_smem : k.uvw.smem(p, bwd);
    OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, (const void*)k.fn) == cudaSuccess) k.regs = attr.numRegs;
    else (void)cudaGetLastError();
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)k.fn, k.uvw.threads, k.smem) != cudaSuccess) {
        (void)cudaGetLastError();
        occ = 1;
    }
    k.ctas_per_sm = std::max(1, k.is_uvw_row ? occ : std::min(occ, 2));
    k.map.ng = 1;
    k.loaded = true;
    return OEQ_OK;
}

// Mirror of oeq::UvwParams (uvw_kernels.cuh).
struct UvwParams {
    const void* X; const void* Y; const void* W; void* Z;
    const void* dZ; void* dX; void* dY; void* dW;
    void* ws;
    long long batch;
    int* status;
    int skip_dw;      // the shared-weight gradient comes from the tensor-core kernel
    int bulk;         // staged rows: all arrays start on a 16-byte boundary
};

// The kernel that a batch takes.
Kernel& uvw_kernel(Kernel& tiled, Kernel& row, const Problem& p, bool bwd, long long batch) {
    if (!row.compiled) return tiled;
    return tiled.compiled && row.loaded && batch > (long long)uvw_row_limit(p, bwd) * row.sm_count ? tiled : row;
}

long long uvw_grid(const Kernel& k, long long batch) {
    const long long tiles = (batch + k.uvw.tile_r - 1) / k.uvw.tile_r;
    return std::max<long long>(1, std::min<long long>((long long)k.sm_count * k.ctas_per_sm, tiles));
}

int load_kernel(Kernel& k, const char* entry, bool want_reduce) {
    if (k.loaded) return OEQ_OK;
    OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, entry));
    if (want_reduce) OEQ_CUDA(cudaLibraryGetKernel(&k.reduce_fn, k.lib, "oeq_reduce_partials"));
    int dev = 0;
    OEQ_CUDA(cudaGetDevice(&dev));
    OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
    int stages = std::min(k.map.max_stages(), env_int("OEQ_B200_STAGES", 4));
    if (k.is_uvu_tc) stages = k.tc_geo.stages;
    if (k.map.slice_warps) stages = k.map.slice_stages;
    if (stages < 2) return fail(OEQ_ERR_UNSUPPORTED, "not enough shared memory for two stages");
    k.stages = stages;
    k.smem = k.map.slice_warps ? k.map.slice_smem : (k.is_uvu_tc ? k.tc_geo.smem : k.map.smem(stages));
    OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, (const void*)k.fn) == cudaSuccess) k.regs = attr.numRegs;
    else (void)cudaGetLastError();
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, (const void*)k.fn, k.threads(), k.smem) != cudaSuccess) {
        (void)cudaGetLastError();
        occ = 1;
    }
    k.ctas_per_sm = std::max(1, std::min(occ, env_int("OEQ_B200_CTAS_PER_SM", 4)));
    if (k.is_uvu_tc) k.ctas_per_sm = 1;
    k.loaded = true;
    return OEQ_OK;
}

// Mirror of oeq::UvuParams (uvu_kernels.cuh).
struct UvuParams {
    const void* X; const void* Y; const void* W; void* Z;
    const void* dZ; void* dX; void* dY; void* dW;
    const long long* rows; const long long* cols; const long long* perm;
    long long n_items, n_nodes;
    void* ws;
    int* status;
    int stages, flags, chunk;
    long long e_lo, e_hi;
    const long long* sum_cols; const long long* sum_perm; const void* sum_ws;
    long long sum_items, sum_e_lo, sum_e_hi;
    int sum_first, sum_chunk;
    const void* EX; const void* EY; const void* EW;
};

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int launch_uvu(Kernel& k, const Problem& p, UvuParams& prm, cudaStream_t stream, int extra_flags = 0,
               long long max_ctas = 0, long long* ctas_out = nullptr, int clear_flags = 0) {
    const int e = p.elem();
    int flags = 0;
    if ((p.x_dim * e) % 16 == 0 && aligned16(prm.X)) flags |= 1;
    // (with several edges per item a bulk copy covers a run of rows: the run has to be a 16-byte multiple)
    const int epi = k.map.epi;
    if ((p.y_dim * e * epi) % 16 == 0 && aligned16(prm.Y)) flags |= 2;
    if (!p.shared && !p.unit && (p.w_numel * e * epi) % 16 == 0 && aligned16(prm.W)) flags |= 4;
    const void* zlike = prm.dZ ? prm.dZ : prm.Z;
    if ((p.z_dim * e) % 16 == 0 && aligned16(zlike)) flags |= 8;
    if (env_int("OEQ_B200_NO_BULK", 0)) flags = 0;
    flags &= ~clear_flags;
    {
        // short rows: 16-byte cp.async from all lanes instead of one bulk copy issued by one lane
        const int limit = env_int("OEQ_B200_VEC_COPY_BYTES", 0);
        const int row_bytes[4] = {p.x_dim * e, p.y_dim * e, p.w_numel * e, p.z_dim * e};
        for (int a = 0; a < 4; ++a)
            if ((flags & (1 << a)) && row_bytes[a] <= limit) flags = (flags & ~(1 << a)) | (256 << a);
    }
    prm.flags = flags | extra_flags;
    prm.stages = k.stages;
    long long want = (prm.n_items + k.map.ng - 1) / k.map.ng;
    long long grid = std::max<long long>(1, std::min<long long>((long long)k.sm_count * k.ctas_per_sm, want));
    if (max_ctas > 0) grid = std::min(grid, max_ctas);     // a caller with bounded scratch narrows the launch
    if (ctas_out) *ctas_out = grid;
    // chunks of consecutive edges are dealt round-robin to the groups: 128 edges unless that leaves a group fewer
    // than eight chunks (the last round then idles a large part of the machine)
    int chunk = env_int("OEQ_B200_CHUNK", 0);
    if (chunk <= 0) {
        chunk = 128;
        const long long groups = grid * k.map.ng;
        while (chunk > k.map.chunk_floor && prm.n_items / (groups * chunk) < 8) chunk /= 2;
        // A short list: smaller chunks while groups would be left without one.  Deterministic walks, whose chunks move to
        // the next boundary (two dependent index reads) or meet a receiver's dZ anew, wait until three in seven would be:
        // 64x0e+32x1o, 59 k edges, forward 137 us with chunks of 32 (as many as groups), 111 with 64; 20 k edges 68 with 32,
        // 63 with 16; 32x(0e..3o) FP64 backward, 6 k edges, 162 with 8, 109 with 16 (forward 131 and 148).
        const bool aligned = prm.rows && (k.map.chunk_floor > 32 || prm.ws);
        while (chunk > 8 && (aligned ? prm.n_items * 7 / 4 : prm.n_items) < groups * chunk) chunk /= 2;
    }
    prm.chunk = std::max(1, chunk);
    void* args[] = {&prm};
    OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)grid), dim3((unsigned)k.threads()), args,
                              (size_t)k.smem, stream));
    return OEQ_OK;
}

// Edges per chunk and CTAs of a slice kernel.  Node rows that fit in L2 are gathered from there whatever the order:
// each walker then takes one run of the edge list (at least 8 edges), which needs its ends aligned once.  Larger graphs
// are dealt in chunks of 128 edges, so that the walkers stay in one neighbourhood of the list.  A walk that adds to the
// rows it gathers (`adds_mb` > 0, atomic backward) has both in L2, up to that many MB.  FP64, whose additions are by eight
// bytes, 32x(0e+1o+2e): one run each / chunks of 128, 10 000 nodes (2 x 23 MB) 476 / 466 us, 15 000 822 / 769, 20 000
// 1187 / 1002; 128x(0e+1o+2e), 3 000 nodes (2 x 28 MB) 771 / 874.  FP32: 32x(0e+1o+2e), 40 000 nodes (2 x 46 MB) 1006 / 1054;
// 128x(0e+1o+2e), 20 000 nodes (2 x 92 MB) 2817 / 2696.
void slice_launch_shape(const Kernel& k, long long edges, size_t gathered_bytes, int adds_mb, long long& grid, int& chunk) {
    const int per_cta = k.map.slice_warps / k.map.n_slice;
    const long long most = (long long)k.sm_count * k.ctas_per_sm;
    const long long walkers = most * per_cta;
    const bool runs = adds_mb ? 2 * gathered_bytes <= ((size_t)adds_mb << 20) : gathered_bytes <= (48u << 20) || edges < walkers * 512;
    chunk = env_int("OEQ_B200_CHUNK", 0);
    if (chunk <= 0) {
        chunk = 128;
        if (runs || edges < walkers * chunk) chunk = (int)std::max<long long>(8, (edges + walkers - 1) / walkers);
    }
    const long long chunks = (edges + chunk - 1) / chunk;
    grid = std::max<long long>(1, std::min(most, (chunks + per_cta - 1) / per_cta));
}

// Row sum: a warp takes a chunk of the sender-ordered edge list and 512 bytes (rows of 8 KB and more: 2 KB) of the rows.  64 edges per chunk, fewer
// when that would leave warps idle.
constexpr int SUM_WARPS_PER_SM = 48;
long long row_sum_blocks(const Problem& p) {
    const int row = pad16(p.x_dim * p.elem()), piece = (row + 511) / 512 >= 16 ? 2048 : 512;
    return (row + piece - 1) / piece;
}
int row_sum_chunk(const Kernel& k, const Problem& p, long long edges) {
    int chunk = env_int("OEQ_B200_SUM_CHUNK", 0);
    if (chunk > 0) return chunk;
    chunk = 64;
    while (chunk > 8 && edges * row_sum_blocks(p) < (long long)chunk * k.sm_count * SUM_WARPS_PER_SM) chunk /= 2;
    return chunk;
}
long long row_sum_grid(const Kernel& k, const Problem& p, long long edges, int chunk) {
    const long long warps = (edges + chunk - 1) / chunk * row_sum_blocks(p);
    return std::max<long long>(1, std::min<long long>((long long)k.sm_count * (SUM_WARPS_PER_SM / 8), (warps + 7) / 8));
}

int launch_slice(Kernel& k, const Problem& p, UvuParams& prm, cudaStream_t stream, int clear_flags = 0) {
    const int e = p.elem();
    const bool full = k.map.slice_full;
    int flags = 0;
    if ((full || (p.x_dim * e) % 16 == 0) && aligned16(prm.X)) flags |= 1;
    if ((full || (p.w_numel * e) % 16 == 0) && aligned16(prm.W)) flags |= 4;
    // rows out: Z by output irrep; dX, or the scratch rows (16-byte aligned with the same pitch)
    if (prm.dX ? ((full || (p.x_dim * e) % 16 == 0) && aligned16(prm.ws ? prm.ws : prm.dX)) : aligned16(prm.Z)) flags |= 8;
    prm.flags = flags & ~clear_flags;
    long long grid = 1;
    slice_launch_shape(k, prm.n_items, (size_t)prm.n_nodes * p.x_dim * e, prm.dX && !prm.ws ? (e == 8 ? 64 : 128) : 0, grid, prm.chunk);
    void* args[] = {&prm};
    OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)grid), dim3((unsigned)k.threads()), args, (size_t)k.smem, stream));
    return OEQ_OK;
}

long long uvu_grid(const Kernel& k, long long n_items) {
    long long want = (n_items + k.map.ng - 1) / k.map.ng;
    return std::max<long long>(1, std::min<long long>((long long)k.sm_count * k.ctas_per_sm, want));
}

}  // namespace

// ====================================================================== C ABI

struct oeq_tp {
    std::mutex mutex;           // a call that launches (and loads kernels the first time) at a time
    Problem prob;
    Kernel fwd, bwd;
    Kernel fwd_row, bwd_row;    // 'uvw' with per-row weights: one row per CTA (then fwd / bwd are for the batches of uvw_row_limit, if any)
    Kernel fwd_ts;              // tensor-core forward ('uvw', shared FP32 weights) with the weights in tensor memory
    bool has_ts = false;
    int ts_smem = 0;
    Kernel fwd_tc;              // the same with the weights in shared memory, for wider problems
    bool has_tc = false;
    Kernel bwd_dw_tc;           // tensor-core weight gradient of the same class of problems
    Kernel bwd_dw_ts;           // the same from rows formed a batch row per lane
    bool has_bwd_tc = false, has_dw_ts = false, has_dw_tc = false;          // either; which
    int dw_smem = 0, dw_threads = 0, dw_ts_smem = 0;
    DwChoice dw_choice;
    // dX and dY of the same class of problems: dT = W dZ on the tensor cores, then the channel-wise backward pass
    Problem grad_product, grad_channels;
    Kernel grad_product_k, grad_channels_k;
    TcGeometry grad_tc;
    bool has_grad_tc = false;
    void* d_packed_t = nullptr; // the transposed weights, split and swizzled (calls whose workspace does not hold them)
    cudaKernel_t pack_t_fn = nullptr;
    Kernel gemm, gemm_dw;       // FP64 with shared weights: the product and the weight gradient as GEMMs
    bool has_gemm = false, has_gemm_bwd = false;
    Kernel dbl;                 // one-pass second derivatives ('uvu', per-row weights)
    bool has_dbl = false;
    TcGeometry tc;
    void* d_packed = nullptr;   // weights split and swizzled for the tensor cores (calls without a workspace)
    cudaKernel_t pack_fn = nullptr;
    int* d_status = nullptr;
    cudaStream_t last_stream = nullptr;
};
struct oeq_conv {
    std::mutex mutex;           // a call that launches (and loads kernels the first time) at a time
    Problem prob;
    bool deterministic = false;
    Kernel fwd, bwd;
    Kernel fwd_tc;              // tensor-core forward pass, when the problem qualifies
    bool has_fwd_tc = false;
    Kernel fwd_slice, bwd_slice;    // slice kernels, for the problems that have their shape
    bool has_fwd_slice = false, has_bwd_slice = false;
    Kernel bwd_recv;            // receiver-order backward pass (needs scratch in the deterministic variant)
    bool has_bwd_recv = false;
    cudaKernel_t sum_rows_fn = nullptr, clear_fn = nullptr;
    Kernel dbl_z, dbl_g;        // second derivatives in two launches; compiled at first use
    int dbl_state = 0;          // 0 not tried, 1 ready, -1 not available
    cudaKernel_t dbl_sum_fn = nullptr, dbl_clear_fn = nullptr;
    int last_bwd_launches = 0;  // kernel launches of the most recent oeq_conv_backward
    int* d_status = nullptr;
    cudaStream_t last_stream = nullptr;
};

extern "C" {

const char* oeq_version(void) { return "oeq_b200 0.1 (sm_100a)"; }
const char* oeq_last_error(void) { return g_error.c_str(); }

int oeq_set_kernel_dir(const char* path) {
    if (!path) return fail(OEQ_ERR_INVALID, "null path");
    g_kernel_dir = path;
    return OEQ_OK;
}
int oeq_set_cache_dir(const char* path) {
    if (!path) return fail(OEQ_ERR_INVALID, "null path");
    g_cache_dir = path;
    return OEQ_OK;
}

static int check_conv_problem(const Problem& p) {
    if (p.mode != OEQ_MODE_UVU) return fail(OEQ_ERR_UNSUPPORTED, "fused convolution supports 'uvu' problems only");
    if (p.shared) return fail(OEQ_ERR_UNSUPPORTED, "fused convolution needs per-edge weights (shared_weights=False)");
    // (shared_weights == 2, "every weight is 1", is a per-edge-weight problem without the array)
    for (const Irrep& r : p.in2)
        if (r.mul != 1) return fail(OEQ_ERR_UNSUPPORTED, "fused convolution needs multiplicity 1 for every irrep of the second input");
    return OEQ_OK;
}

int oeq_precompile(const oeq_problem_desc* desc, int kinds) {
    Problem p;
    int rc = ingest(desc, p);
    if (rc) return rc;
    if (p.mode == OEQ_MODE_UVW) {
        if (kinds & 6) return fail(OEQ_ERR_UNSUPPORTED, "fused convolution supports 'uvu' problems only");
        Kernel f, b, fr, br, tc;
        if (uvw_gemm_supported(p)) {
            Problem pp, pc;
            Kernel dw, kp, kc;
            if ((rc = build_uvw_gemm(p, K_UVW_GEMM, f))) return rc;
            rc = build_uvw_gemm_backward(p, pp, pc, dw, kp, kc);
            if (rc && rc != OEQ_ERR_UNSUPPORTED) return rc;
            if (gemm_keeps_tiled(p) && (rc = build_tp(p, false, fr, fr))) return rc;
        } else if ((rc = build_tp(p, false, f, fr))) {
            return rc;
        }
        if ((rc = build_tp(p, true, b, br))) return rc;
        TcGeometry g;
        int smem = 0, threads = 0;
        if (uvw_ts_geometry(p, smem) && uvw_ts_faster(p)) rc = build_uvw_ts(p, tc);
        else if (uvw_tc_geometry(p, g)) rc = build_uvw_tc(p, g, tc);
        if (rc) return rc;
        Kernel dw, product, channels;
        if (uvw_tc_dw_geometry(p, smem, threads)) {
            const DwChoice choice = uvw_dw_choice(p);
            const bool ts = uvw_ts_dw_geometry(p, smem);
            Kernel wider;
            if ((ts && (rc = build_uvw_ts_dw(p, dw))) || ((!ts || choice.few || choice.many) && (rc = build_uvw_tc_bwd(p, K_UVW_TC_DW, wider)))) return rc;
            Problem pp, pc;
            rc = build_uvw_gradients(p, pp, pc, g, product, channels);
            if (rc && rc != OEQ_ERR_UNSUPPORTED) return rc;
        }
        return OEQ_OK;
    }
    auto one = [&](int kind) {
        Kernel k;
        return build_uvu(p, kind, k);
    };
    if (kinds & 1) {
        if ((rc = one(K_FWD_BATCH)) || (rc = one(K_BWD_BATCH))) return rc;
        if (double_backward_supported(p)) {
            Kernel k;
            rc = build_uvu_dbl(p, k);
            if (rc && rc != OEQ_ERR_UNSUPPORTED) return rc;
        }
    }
    if (kinds & 6) {
        if ((rc = check_conv_problem(p))) return rc;
    }
    UvuTcGeometry geo;
    const bool tc = (kinds & 6) && uvu_tc_geometry(p, geo);
    const bool recv = (kinds & 6) && recv_backward_supported(p);
    for (int det = 1; det >= 0; --det) {
        if (!(kinds & (det ? 2 : 4))) continue;
        Kernel f, b, k, kr;
        const int rf = build_slice_fwd(p, det != 0, f), rb = build_slice_bwd(p, det != 0, b);
        if (rf && rf != OEQ_ERR_UNSUPPORTED) return rf;
        if (rb && rb != OEQ_ERR_UNSUPPORTED) return rb;
        if ((rf || group_forward_beside_slice(p, f)) && (rc = one(det ? K_FWD_DET : K_FWD_ATOMIC))) return rc;
        if ((rc = one(det ? K_BWD_DET : K_BWD_ATOMIC))) return rc;
        if (tc && (rc = build_uvu_tc(p, det != 0, k))) return rc;
        if (recv && recv_beside_slice(p, !rb, b, det != 0) && (rc = build_uvu_recv(p, det != 0, kr))) return rc;
    }
    if ((kinds & 8) && (kinds & 6) && conv_second_possible(p)) {
        for (int det = 0; det < 2; ++det) {
            if (!(kinds & (det ? 2 : 4))) continue;
            Kernel z, g;
            rc = build_conv_dbl(p, det != 0, z, g);
            if (rc && rc != OEQ_ERR_UNSUPPORTED) return rc;
        }
    }
    return OEQ_OK;
}

// ---------------------------------------------------------------- batch TP

int oeq_tp_create(const oeq_problem_desc* desc, oeq_tp** out) {
    if (!out) return fail(OEQ_ERR_INVALID, "null output handle");
    *out = nullptr;
    oeq_tp* h = new oeq_tp();
    int rc = ingest(desc, h->prob);
    if (!rc && uvw_gemm_supported(h->prob)) {
        rc = build_uvw_gemm(h->prob, K_UVW_GEMM, h->gemm);
        h->has_gemm = rc == OEQ_OK;
        if (!rc) {
            const int rc2 = build_uvw_gemm_backward(h->prob, h->grad_product, h->grad_channels, h->gemm_dw, h->grad_product_k, h->grad_channels_k);
            h->has_gemm_bwd = rc2 == OEQ_OK;
            if (rc2 != OEQ_OK && rc2 != OEQ_ERR_UNSUPPORTED) rc = rc2;
        }
    }
    if (!rc && (!h->has_gemm || gemm_keeps_tiled(h->prob))) rc = build_tp(h->prob, false, h->fwd, h->fwd_row);
    if (!rc) rc = build_tp(h->prob, true, h->bwd, h->bwd_row);
    if (!rc && uvw_ts_geometry(h->prob, h->ts_smem) && uvw_ts_faster(h->prob)) {
        rc = build_uvw_ts(h->prob, h->fwd_ts);
        h->has_ts = rc == OEQ_OK;
    } else if (!rc && uvw_tc_geometry(h->prob, h->tc)) {
        rc = build_uvw_tc(h->prob, h->tc, h->fwd_tc);
        h->has_tc = rc == OEQ_OK;
    }
    if (!rc && uvw_tc_dw_geometry(h->prob, h->dw_smem, h->dw_threads)) {
        h->dw_choice = uvw_dw_choice(h->prob);
        h->has_dw_ts = uvw_ts_dw_geometry(h->prob, h->dw_ts_smem);
        h->has_dw_tc = !h->has_dw_ts || h->dw_choice.few || h->dw_choice.many;
        if (h->has_dw_ts) rc = build_uvw_ts_dw(h->prob, h->bwd_dw_ts);
        if (!rc && h->has_dw_tc) rc = build_uvw_tc_bwd(h->prob, K_UVW_TC_DW, h->bwd_dw_tc);
        h->has_bwd_tc = rc == OEQ_OK;
        if (!rc) {
            const int rc2 = build_uvw_gradients(h->prob, h->grad_product, h->grad_channels, h->grad_tc, h->grad_product_k, h->grad_channels_k);
            h->has_grad_tc = rc2 == OEQ_OK;
            if (rc2 != OEQ_OK && rc2 != OEQ_ERR_UNSUPPORTED) rc = rc2;
        }
    }
    if (!rc && double_backward_supported(h->prob)) {
        const int rc2 = build_uvu_dbl(h->prob, h->dbl);
        if (rc2 == OEQ_OK) h->has_dbl = true;
        else if (rc2 != OEQ_ERR_UNSUPPORTED) rc = rc2;
    }
    if (rc) {
        delete h;
        return rc;
    }
    *out = h;
    return OEQ_OK;
}

int oeq_tp_destroy(oeq_tp* h) {
    if (!h) return OEQ_OK;
    if (h->d_status) cudaFree(h->d_status);
    if (h->d_packed) cudaFree(h->d_packed);
    if (h->d_packed_t) cudaFree(h->d_packed_t);
    for (Kernel* k : {&h->fwd, &h->bwd, &h->fwd_row, &h->bwd_row, &h->fwd_ts, &h->fwd_tc, &h->bwd_dw_tc, &h->bwd_dw_ts, &h->grad_product_k, &h->grad_channels_k, &h->gemm, &h->gemm_dw, &h->dbl})
        if (k->lib) cudaLibraryUnload(k->lib);
    delete h;
    return OEQ_OK;
}

int64_t oeq_tp_weight_numel(const oeq_tp* h) { return h ? h->prob.w_numel : -1; }

static int ensure_status(int** d_status) {
    if (*d_status) return OEQ_OK;
    OEQ_CUDA(cudaMalloc(d_status, sizeof(int)));
    OEQ_CUDA(cudaMemset(*d_status, 0, sizeof(int)));
    return OEQ_OK;
}

// Weights in the operand layout: at `workspace` when it holds them, else in memory of the handle's own (`own`), which
// every call that has no workspace writes anew: such calls are for one stream at a time.
static int packed_weights(const TcGeometry& geo, void* workspace, size_t workspace_bytes, void*& own, void*& packed) {
    packed = workspace;
    if (workspace && workspace_bytes >= geo.packed_bytes && aligned16(workspace)) return OEQ_OK;
    if (!own) OEQ_CUDA(cudaMalloc(&own, geo.packed_bytes));
    packed = own;
    return OEQ_OK;
}

static int load_uvw_tc(Kernel& k, const TcGeometry& geo, cudaKernel_t& pack) {
    if (k.loaded) return OEQ_OK;
    OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, "oeq_uvw_tc_kernel"));
    OEQ_CUDA(cudaLibraryGetKernel(&pack, k.lib, "oeq_uvw_pack_weights"));
    int dev = 0;
    OEQ_CUDA(cudaGetDevice(&dev));
    OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
    k.smem = geo.smem;
    OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, (const void*)k.fn) == cudaSuccess) k.regs = attr.numRegs;
    else (void)cudaGetLastError();
    k.loaded = true;
    return OEQ_OK;
}

static int launch_uvw_ts(Kernel& k, int smem, const Problem& p, long long batch, const void* X, const void* Y, const void* W, void* Z, int* status, cudaStream_t st) {
    if (!k.loaded) {
        OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
        OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, "oeq_uvw_ts_kernel"));
        int dev = 0;
        OEQ_CUDA(cudaGetDevice(&dev));
        OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
        k.smem = smem;
        OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
        cudaFuncAttributes attr;
        if (cudaFuncGetAttributes(&attr, (const void*)k.fn) == cudaSuccess) k.regs = attr.numRegs;
        else (void)cudaGetLastError();
        k.loaded = true;
    }
    struct { const void* X; const void* Y; const void* W; void* Z; long long batch; int* status; int in_vec, z_vec; }
        tp{X, Y, W, Z, batch, status, aligned16(X) && aligned16(Y), aligned16(Z)};
    void* args[] = {&tp};
    const long long tiles = (batch + TS_ROWS - 1) / TS_ROWS * (long long)p.out.size();
    OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)std::min<long long>(k.sm_count, tiles)), dim3(TS_THREADS), args, (size_t)k.smem, st));
    return OEQ_OK;
}

// `pack`: the weights have to be brought into the operand layout first (once per call).
static int launch_uvw_tc(Kernel& k, const TcGeometry& geo, cudaKernel_t pack_fn, void* packed, bool pack, long long batch, const void* X, const void* Y,
                         const void* W, void* Z, int* status, cudaStream_t st) {
    if (pack) {
        void* args[] = {(void*)&W, &packed};
        OEQ_CUDA(cudaLaunchKernel((const void*)pack_fn, dim3(16, geo.paths), dim3(256), args, 0, st));
    }
    struct { const void* X; const void* Y; const void* Wp; void* Z; long long batch; int* status; int dealt; unsigned long long* prof; }
        tp{X, Y, packed, Z, batch, status, 0, nullptr};
    void* args[] = {&tp};
    // Up to a chunk per CTA and output: output irreps over the grid's y dimension.  Then, up to some rows per SM, chunks of
    // all outputs dealt; above, a share of the rows each, whose balance does not depend on the costs that the deal assumes.
    // Shares / dealt in us, forward and W dZ: 64x(0e+1o+2e), 8 000 rows 72 / 58 and 43 / 35, 16 000 98 / 98 and 60 / 58, 24 000
    // 139 / 136 and 85 / 82, 26 000 146 / 146 and 90 / 91, 29 600 156 / 166 and 97 / 101; 32x(0e+1o+2e), 29 600 77 / 73 and
    // 52 / 52.
    long long grid = std::max<long long>(1, std::min<long long>(k.sm_count, (batch + 23) / 24));
    const unsigned split = grid * geo.outputs <= k.sm_count ? geo.outputs : 1;
    if (split == 1 && geo.outputs > 1 && batch <= (long long)geo.dealt_rows_per_sm * k.sm_count) {
        tp.dealt = 1;
        grid = k.sm_count;
    }
#ifdef OEQ_DEV_PROFILE
    if (env_int("OEQ_B200_TC_PROFILE", 0)) {
        // cycle accounting of the roles of CTA 0 (development aid): synchronous, prints to stderr
        OEQ_CUDA(cudaMalloc(&tp.prof, 32 * 8));
        OEQ_CUDA(cudaMemsetAsync(tp.prof, 0, 32 * 8, st));
        OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)grid, split), dim3((unsigned)geo.threads()), args, (size_t)k.smem, st));
        unsigned long long hb[32];
        OEQ_CUDA(cudaMemcpyAsync(hb, tp.prof, sizeof hb, cudaMemcpyDeviceToHost, st));
        OEQ_CUDA(cudaStreamSynchronize(st));
        cudaFree(tp.prof);
        fprintf(stderr, "[oeq_b200 uvw tc profile] mma: wait %llu issue %llu | epilogue: tiles %llu wait %llu drain %llu\n", hb[8], hb[9],
                hb[18], hb[16], hb[17]);
        return OEQ_OK;
    }
#endif
    OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)grid, split), dim3((unsigned)geo.threads()), args, (size_t)k.smem, st));
    return OEQ_OK;
}

// Mirror of oeq::UvwGemmParams (uvw_gemm_kernels.cuh).
struct UvwGemmParams {
    const void* X; const void* Y; const void* W; const void* dZ;
    void* Z; void* ws;
    long long batch;
    int shares;
};

static int load_gemm(Kernel& k) {
    if (k.loaded) return OEQ_OK;
    OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
    OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, "oeq_uvw_gemm_kernel"));
    OEQ_CUDA(cudaLibraryGetKernel(&k.reduce_fn, k.lib, "oeq_reduce_partials"));
    int dev = 0;
    OEQ_CUDA(cudaGetDevice(&dev));
    OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
    k.smem = GEMM_SMEM;
    OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, (const void*)k.fn) == cudaSuccess) k.regs = attr.numRegs;
    else (void)cudaGetLastError();
    k.loaded = true;
    return OEQ_OK;
}

// Z (or dT) = the product of problem `p` over `batch` rows.
static int launch_gemm(Kernel& k, const Problem& p, long long batch, const void* X, const void* Y, const void* W, void* Z, cudaStream_t st) {
    int rc = load_gemm(k);
    if (rc) return rc;
    UvwGemmParams prm{X, Y, W, nullptr, Z, nullptr, batch, 1};
    int y = 0, rows = GEMM_TILE;
    for (const Irrep& r : p.out) {
        y += (r.mul + GEMM_TILE - 1) / GEMM_TILE;
        rows = std::min(rows, GEMM_TILE / r.dim);
    }
    void* args[] = {&prm};
    OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)((batch + rows - 1) / rows), (unsigned)y), dim3(256), args, (size_t)k.smem, st));
    return OEQ_OK;
}

size_t oeq_tp_forward_workspace_bytes(const oeq_tp* h) { return h && h->has_tc ? h->tc.packed_bytes : 0; }

int oeq_tp_forward(oeq_tp* h, int64_t batch, const void* X, const void* Y, const void* W, void* Z, void* stream) {
    return oeq_tp_forward_ws(h, batch, X, Y, W, Z, nullptr, 0, stream);
}

int oeq_tp_forward_ws(oeq_tp* h, int64_t batch, const void* X, const void* Y, const void* W, void* Z, void* workspace, size_t workspace_bytes,
                      void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (batch < 0) return fail(OEQ_ERR_INVALID, "negative batch");
    if (batch == 0) return OEQ_OK;
    if (!X || !Y || !W || !Z) return fail(OEQ_ERR_INVALID, "null buffer");
    int rc = ensure_status(&h->d_status);
    if (rc) return rc;
    h->last_stream = (cudaStream_t)stream;
    if (h->has_ts) return launch_uvw_ts(h->fwd_ts, h->ts_smem, h->prob, batch, X, Y, W, Z, h->d_status, (cudaStream_t)stream);
    if (h->has_tc) {
        void* packed = nullptr;
        if ((rc = load_uvw_tc(h->fwd_tc, h->tc, h->pack_fn)) || (rc = packed_weights(h->tc, workspace, workspace_bytes, h->d_packed, packed)))
            return rc;
        return launch_uvw_tc(h->fwd_tc, h->tc, h->pack_fn, packed, true, batch, X, Y, W, Z, h->d_status, (cudaStream_t)stream);
    }
    if (h->has_gemm) {
        if ((rc = load_gemm(h->gemm))) return rc;
        if (!h->fwd.compiled || !gemm_forward_tiled(h->prob, batch, h->gemm.sm_count)) return launch_gemm(h->gemm, h->prob, batch, X, Y, W, Z, (cudaStream_t)stream);
    }
    if (h->prob.mode == OEQ_MODE_UVW) {
        if (h->fwd_row.compiled && (rc = load_uvw(h->fwd_row, h->prob, false))) return rc;
        Kernel& k = uvw_kernel(h->fwd, h->fwd_row, h->prob, false, batch);
        if ((rc = load_uvw(k, h->prob, false))) return rc;
        UvwParams up{};
        up.X = X; up.Y = Y; up.W = W; up.Z = Z; up.batch = batch; up.status = h->d_status;
        up.bulk = aligned16(X) && aligned16(Y) && aligned16(W);
        void* args[] = {&up};
        OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)uvw_grid(k, batch)), dim3((unsigned)k.uvw.threads), args, (size_t)k.smem,
                                  (cudaStream_t)stream));
        return OEQ_OK;
    }
    if ((rc = load_kernel(h->fwd, "oeq_uvu_kernel", false))) return rc;
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.Z = Z;
    prm.n_items = batch; prm.n_nodes = batch; prm.status = h->d_status;
    return launch_uvu(h->fwd, h->prob, prm, (cudaStream_t)stream);
}

size_t oeq_tp_workspace_bytes(const oeq_tp* h, int64_t batch) {
    if (!h || !h->prob.shared || batch <= 0) return 0;
    // one partial weight gradient per group (uvu) or per CTA (uvw) of the backward launch; sized for the
    // largest grid the launch can use on any device (256 SMs)
    long long groups;
    if (h->prob.mode == OEQ_MODE_UVW) {
        const long long tiles = (batch + h->bwd.uvw.tile_r - 1) / h->bwd.uvw.tile_r;
        groups = std::max<long long>(std::min<long long>(tiles, 256ll * 2), h->has_bwd_tc ? 256ll : 0ll);
    } else {
        groups = 256ll * 4 * h->bwd.map.ng;
    }
    if (h->has_gemm_bwd) {
        const size_t partial = (size_t)h->prob.w_numel * 8, tiled = gemm_backward_tiled(h->prob, batch, 256) ? (size_t)groups * partial : 0;
        return std::max({(size_t)gemm_shares(h->prob, batch, 256) * partial, tiled, std::min((size_t)batch * h->grad_product.z_dim * 8, UVW_DT_BYTES)});
    }
    size_t bytes = (size_t)groups * h->prob.w_numel * h->prob.elem();
    if (h->has_grad_tc) bytes = std::max(bytes, std::min((size_t)batch * h->grad_product.z_dim * 4, UVW_DT_BYTES) + h->grad_tc.packed_bytes + 256);
    return bytes;
}

int oeq_tp_backward(oeq_tp* h, int64_t batch, const void* X, const void* Y, const void* W, const void* dZ, void* dX,
                    void* dY, void* dW, void* workspace, size_t workspace_bytes, void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (batch < 0) return fail(OEQ_ERR_INVALID, "negative batch");
    cudaStream_t st = (cudaStream_t)stream;
    const Problem& p = h->prob;
    if (batch == 0) {
        if (p.shared && dW) OEQ_CUDA(cudaMemsetAsync(dW, 0, (size_t)p.w_numel * p.elem(), st));
        return OEQ_OK;
    }
    if (!X || !Y || !W || !dZ || !dX || !dY || !dW) return fail(OEQ_ERR_INVALID, "null buffer");
    int rc = ensure_status(&h->d_status);
    if (rc) return rc;
    // dX and dY of a shared-weight problem from dT rows in the workspace (blocks of the batch when they do not all fit)
    auto gradients_from_dt = [&](long long block, auto&& product) -> int {
        const size_t e = p.elem();
        int r = load_kernel(h->grad_channels_k, "oeq_uvu_kernel", false);
        for (long long b0 = 0; b0 < batch && !r; b0 += block) {
            const long long rows = std::min<long long>(block, batch - b0);
            if ((r = product(b0, rows, (const char*)dZ + (size_t)b0 * p.z_dim * e))) break;
            UvuParams prm{};
            prm.X = (const char*)X + (size_t)b0 * p.x_dim * e;
            prm.Y = (const char*)Y + (size_t)b0 * p.y_dim * e;
            prm.dZ = workspace;
            prm.dX = (char*)dX + (size_t)b0 * p.x_dim * e;
            prm.dY = (char*)dY + (size_t)b0 * p.y_dim * e;
            prm.n_items = rows; prm.n_nodes = rows; prm.status = h->d_status;
            r = launch_uvu(h->grad_channels_k, h->grad_channels, prm, st);
        }
        return r;
    };
    // (a workspace that does not hold a partial gradient and a dT row each, 16-byte aligned, is for the tiled kernel)
    const size_t wbytes = (size_t)p.w_numel * 8, dt_row = (size_t)h->grad_product.z_dim * 8;
    if (h->has_gemm_bwd && (rc = load_gemm(h->gemm_dw))) return rc;
    const bool gemm_tiled = h->has_gemm_bwd && gemm_backward_tiled(p, batch, h->gemm_dw.sm_count) &&
                            workspace_bytes / wbytes >= (size_t)std::min<long long>((batch + h->bwd.uvw.tile_r - 1) / h->bwd.uvw.tile_r, 2ll * h->gemm_dw.sm_count);
    if (h->has_gemm_bwd && workspace && aligned16(workspace) && workspace_bytes >= std::max(wbytes, dt_row) && !gemm_tiled) {
        const long long block = (long long)std::min<size_t>((size_t)batch, workspace_bytes / dt_row);
        h->last_stream = st;
        Kernel& k = h->gemm_dw;
        long long shares = std::min<long long>(gemm_shares(p, batch, k.sm_count), (long long)(workspace_bytes / wbytes));
        int tiles = 0, n = p.w_numel;
        for (const Instr& t : p.instr)
            tiles += ((p.in1[t.i1].mul + GEMM_TILE - 1) / GEMM_TILE) * ((p.out[t.io].mul + GEMM_TILE - 1) / GEMM_TILE);
        UvwGemmParams prm{X, Y, nullptr, dZ, nullptr, shares == 1 ? dW : workspace, batch, (int)shares};
        void* args[] = {&prm};
        OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)shares, (unsigned)tiles), dim3(256), args, (size_t)k.smem, st));
        if (shares > 1) {
            const void* ws = workspace;
            void* rargs[] = {&ws, &dW, &n, &shares};
            OEQ_CUDA(cudaLaunchKernel((const void*)k.reduce_fn, dim3((n + 31) / 32), dim3(256), rargs, 0, st));
        }
        return gradients_from_dt(block, [&](long long, long long rows, const void* dz) {
            return launch_gemm(h->grad_product_k, h->grad_product, rows, dz, nullptr, W, workspace, st);
        });
    }
    if (p.mode == OEQ_MODE_UVW) {
        if (h->bwd_row.compiled && (rc = load_uvw(h->bwd_row, p, true))) return rc;
        Kernel& main = uvw_kernel(h->bwd, h->bwd_row, p, true, batch);
        if ((rc = load_uvw(main, p, true))) return rc;
        long long ctas = uvw_grid(main, batch);
        if (p.shared) {
            const size_t need = (size_t)ctas * p.w_numel * p.elem();
            if (!workspace || workspace_bytes < need)
                return fail(OEQ_ERR_INVALID, "workspace too small for the shared-weight gradient (see oeq_tp_workspace_bytes)");
        }
        UvwParams up{};
        up.X = X; up.Y = Y; up.W = W; up.dZ = dZ; up.dX = dX; up.dY = dY; up.dW = dW; up.ws = workspace;
        up.batch = batch; up.status = h->d_status;
        up.bulk = aligned16(X) && aligned16(Y) && aligned16(W) && aligned16(dZ) && aligned16(dW);
        h->last_stream = st;
        if (h->has_bwd_tc) {
            // weight gradient on the tensor cores (per-CTA partial sums in the workspace, then the fixed-order
            // reduction); the FMA kernel computes dX and dY only
            const bool ts = h->has_dw_ts && !(h->has_dw_tc && h->dw_choice.wider(batch, main.sm_count));
            Kernel& k = ts ? h->bwd_dw_ts : h->bwd_dw_tc;
            if (!k.loaded) {
                OEQ_CUDA(cudaLibraryLoadData(&k.lib, k.code.cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0));
                OEQ_CUDA(cudaLibraryGetKernel(&k.fn, k.lib, ts ? "oeq_uvw_ts_dw_kernel" : "oeq_uvw_tc_dw_kernel"));
                OEQ_CUDA(cudaLibraryGetKernel(&k.reduce_fn, k.lib, ts ? "oeq_ts_reduce" : "oeq_reduce_partials"));
                int dev = 0;
                OEQ_CUDA(cudaGetDevice(&dev));
                OEQ_CUDA(cudaDeviceGetAttribute(&k.sm_count, cudaDevAttrMultiProcessorCount, dev));
                k.smem = ts ? h->dw_ts_smem : h->dw_smem;
                OEQ_CUDA(cudaFuncSetAttribute((const void*)k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
                k.loaded = true;
            }
            if (ts) {
                const long long tiles = (batch + TG_ROWS - 1) / TG_ROWS * (long long)p.out.size();
                // (the CTAs, and with them the order of the sums, do not depend on the workspace: an output has no more of them than the
                // least workspace that a call may come with holds partial gradients; with a CTA per tile, one output, 32x2e with 0e took
                // 10.5 us up to 800 rows, with half as many 12.4)
                int most = (int)std::max(ctas, h->dw_choice.wider_ctas(batch, k.sm_count)), all = (int)std::min<long long>(k.sm_count, tiles);
                if ((size_t)most * p.w_numel * p.elem() > workspace_bytes)
                    return fail(OEQ_ERR_INVALID, "workspace too small for the shared-weight gradient (see oeq_tp_workspace_bytes)");
                struct { const void* X; const void* Y; const void* dZ; void* ws; long long batch; int* status; int in_vec, most; }
                    tp{X, Y, dZ, workspace, batch, h->d_status, aligned16(X) && aligned16(Y) && aligned16(dZ), most};
                void* targs[] = {&tp};
                OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)all), dim3(TS_THREADS), targs, (size_t)k.smem, st));
                const void* ws = workspace;
                long long rows = batch;
                void* rargs[] = {&ws, &dW, &rows, &all, &most};
                OEQ_CUDA(cudaLaunchKernel((const void*)k.reduce_fn, dim3((p.w_numel + 31) / 32), dim3(256), rargs, 0, st));
            } else {
                long long dw_ctas = h->dw_choice.wider_ctas(batch, k.sm_count);
                if ((size_t)dw_ctas * p.w_numel * p.elem() > workspace_bytes)
                    return fail(OEQ_ERR_INVALID, "workspace too small for the shared-weight gradient (see oeq_tp_workspace_bytes)");
                struct { const void* X; const void* Y; const void* dZ; void* ws; long long batch; int* status; }
                    tp{X, Y, dZ, workspace, batch, h->d_status};
                void* targs[] = {&tp};
                // groups of paths that fill the 128 rows of an MMA (tb_groups in the kernel); few rows: dealt over CTAs
                unsigned dw_groups = h->dw_choice.groups;
                if (dw_ctas * dw_groups > k.sm_count) dw_groups = 1;
                OEQ_CUDA(cudaLaunchKernel((const void*)k.fn, dim3((unsigned)dw_ctas, dw_groups), dim3((unsigned)h->dw_threads), targs, (size_t)k.smem, st));
                int n = p.w_numel;
                const void* ws = workspace;
                void* rargs[] = {&ws, &dW, &n, &dw_ctas};
                OEQ_CUDA(cudaLaunchKernel((const void*)k.reduce_fn, dim3((n + 31) / 32), dim3(256), rargs, 0, st));
            }
            up.skip_dw = 1;
            up.ws = nullptr;
            // dX and dY in two steps over dT rows, which take the partial gradients' place in the workspace
            const size_t row = (size_t)h->grad_product.z_dim * 4, tail = h->grad_tc.packed_bytes;
            // (their weights at the end of the workspace, unless it is too small to hold them beside the rows)
            const size_t least = (size_t)std::min<long long>(batch, 4096) * row;
            const size_t room = workspace_bytes >= least + tail + 256 ? (workspace_bytes - tail) / 256 * 256 : workspace_bytes;
            const long long block = h->has_grad_tc && aligned16(workspace) ? (long long)std::min<size_t>((size_t)batch, room / row) : 0;
            if (block > 0 && (block == batch || block >= 4096)) {
                void* packed = nullptr;
                if ((rc = load_uvw_tc(h->grad_product_k, h->grad_tc, h->pack_t_fn)) ||
                    (rc = packed_weights(h->grad_tc, (char*)workspace + room, workspace_bytes - room, h->d_packed_t, packed)))
                    return rc;
                return gradients_from_dt(block, [&](long long b0, long long rows, const void* dz) {
                    return launch_uvw_tc(h->grad_product_k, h->grad_tc, h->pack_t_fn, packed, b0 == 0, rows, dz, nullptr, W, workspace,
                                         h->d_status, st);
                });
            }
        }
        void* args[] = {&up};
        OEQ_CUDA(cudaLaunchKernel((const void*)main.fn, dim3((unsigned)ctas), dim3((unsigned)main.uvw.threads), args, (size_t)main.smem, st));
        if (p.shared && !h->has_bwd_tc) {
            int n = p.w_numel;
            const void* ws = workspace;
            void* rargs[] = {&ws, &dW, &n, &ctas};
            OEQ_CUDA(cudaLaunchKernel((const void*)h->bwd.reduce_fn, dim3((n + 31) / 32), dim3(256), rargs, 0, st));
        }
        return OEQ_OK;
    }
    if ((rc = load_kernel(h->bwd, "oeq_uvu_kernel", true))) return rc;
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.dZ = dZ; prm.dX = dX; prm.dY = dY; prm.dW = dW;
    prm.n_items = batch; prm.n_nodes = batch; prm.status = h->d_status;
    long long groups = 0;
    if (p.shared) {
        groups = uvu_grid(h->bwd, batch) * h->bwd.map.ng;
        const size_t need = (size_t)groups * p.w_numel * p.elem();
        if (!workspace || workspace_bytes < need)
            return fail(OEQ_ERR_INVALID, "workspace too small for the shared-weight gradient (see oeq_tp_workspace_bytes)");
        prm.ws = workspace;
    }
    h->last_stream = st;
    rc = launch_uvu(h->bwd, p, prm, st);
    if (rc) return rc;
    if (p.shared) {
        int n = p.w_numel;
        const void* ws = workspace;
        void* args[] = {&ws, &dW, &n, &groups};
        OEQ_CUDA(cudaLaunchKernel((const void*)h->bwd.reduce_fn, dim3((n + 31) / 32), dim3(256), args, 0, st));
    }
    return OEQ_OK;
}

int oeq_tp_has_double_backward(const oeq_tp* h) { return h && h->has_dbl ? 1 : 0; }

int oeq_tp_double_backward(oeq_tp* h, int64_t batch, const void* X, const void* Y, const void* W, const void* dZ,
                           const void* EX, const void* EY, const void* EW, void* GX, void* GY, void* GW, void* GdZ,
                           void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (!h->has_dbl) return fail(OEQ_ERR_UNSUPPORTED, "no one-pass second-derivative kernel for this problem: compose it from "
                                                      "oeq_tp_forward and oeq_tp_backward");
    if (batch < 0) return fail(OEQ_ERR_INVALID, "negative batch");
    if (batch == 0) return OEQ_OK;
    if (!X || !Y || !W || !dZ || !EX || !EY || !EW || !GX || !GY || !GW || !GdZ) return fail(OEQ_ERR_INVALID, "null buffer");
    int rc = ensure_status(&h->d_status);
    if (!rc) rc = load_kernel(h->dbl, "oeq_uvu_kernel", false);
    if (rc) return rc;
    const Problem& p = h->prob;
    const int e = p.elem();
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.dZ = dZ; prm.EX = EX; prm.EY = EY; prm.EW = EW;
    prm.dX = GX; prm.dY = GY; prm.dW = GW; prm.Z = GdZ;
    prm.n_items = batch; prm.n_nodes = batch; prm.status = h->d_status;
    h->last_stream = (cudaStream_t)stream;
    // launch_uvu derives the bulk-copy bits from X, Y, W, dZ; a cotangent that breaks the 16-byte rule clears
    // the bit of its pair
    int clear = 0;
    if (!aligned16(EX)) clear |= 1;
    if (!aligned16(EY)) clear |= 2;
    if (!aligned16(EW)) clear |= 4;
    (void)e;
    return launch_uvu(h->dbl, p, prm, (cudaStream_t)stream, 0, 0, nullptr, clear);
}

static int check_status(int* d_status, cudaStream_t st) {
    if (!d_status) return OEQ_OK;
    int v = 0;
    OEQ_CUDA(cudaStreamSynchronize(st));
    OEQ_CUDA(cudaMemcpy(&v, d_status, sizeof v, cudaMemcpyDeviceToHost));
    if (v != 0) {
        cudaMemset(d_status, 0, sizeof v);
        return fail(OEQ_ERR_DEVICE_WAIT, "a kernel abandoned a bounded wait (code " + std::to_string(v) + ")");
    }
    return OEQ_OK;
}
int oeq_tp_check(oeq_tp* h) { return h ? check_status(h->d_status, h->last_stream) : fail(OEQ_ERR_INVALID, "null handle"); }

static int launch_info(const Kernel& k, int* threads, int* ng, int* ps, int* stages, int* smem, int* regs) {
    if (threads) *threads = k.is_uvw ? k.uvw.threads : k.threads();
    if (ng) *ng = k.map.ng;
    if (ps) *ps = k.map.ps;
    if (stages) *stages = k.stages;
    if (smem) *smem = k.smem;
    if (regs) *regs = k.regs;
    return OEQ_OK;
}
int oeq_tp_launch_info(const oeq_tp* h, int which, int* threads, int* ng, int* ps, int* stages, int* smem, int* regs) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    if (!which && h->has_ts) {
        if (threads) *threads = TS_THREADS;
        if (ng) *ng = 1;
        if (ps) *ps = 1;
        if (stages) *stages = TS_STAGES;
        if (smem) *smem = h->fwd_ts.smem;
        if (regs) *regs = h->fwd_ts.regs;
        return OEQ_OK;
    }
    if (!which && h->has_tc) {
        if (threads) *threads = h->tc.threads();
        if (ng) *ng = 1;
        if (ps) *ps = 1;
        if (stages) *stages = 2;
        if (smem) *smem = h->fwd_tc.smem;
        if (regs) *regs = h->fwd_tc.regs;
        return OEQ_OK;
    }
    if (which ? h->has_gemm_bwd : h->has_gemm) return launch_info(which ? h->gemm_dw : h->gemm, threads, ng, ps, stages, smem, regs);
    const Kernel& row = which ? h->bwd_row : h->fwd_row;
    return launch_info(row.compiled ? row : which ? h->bwd : h->fwd, threads, ng, ps, stages, smem, regs);
}

// ---------------------------------------------------------------- backward pass that allocates nothing

// Scratch for oeq_tp_backward_noalloc: lives in the library image, so every GPU that loads the
// library holds these bytes until the process exits.
constexpr size_t NOALLOC_SCRATCH_BYTES = 8u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
// In host code the array's name only stands for the symbol; the device address is looked up
// once per device (with that device current) and remembered here.
static void* g_noalloc_scratch_addr[64] = {nullptr};
static std::mutex g_noalloc_mutex;

static int noalloc_scratch(void** out) {
    int dev = 0;
    OEQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(OEQ_ERR_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);     // two host threads may make a device's first call at once
    if (!g_noalloc_scratch_addr[dev]) {
        void* ptr = nullptr;
        OEQ_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        g_noalloc_scratch_addr[dev] = ptr;
    }
    *out = g_noalloc_scratch_addr[dev];
    return OEQ_OK;
}

int oeq_tp_backward_noalloc(oeq_tp* h, int64_t batch, const void* X, const void* Y, const void* W, const void* dZ,
                            void* dX, void* dY, void* dW, void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    const Problem& p = h->prob;
    if (!p.shared)
        return fail(OEQ_ERR_INVALID, "per-row weights need no scratch: call oeq_tp_backward with a null workspace");
    if (batch <= 0) return fail(OEQ_ERR_INVALID, "batch must be positive");
    if (!X || !Y || !W || !dZ || !dX || !dY || !dW) return fail(OEQ_ERR_INVALID, "null buffer");
    const size_t slice = (size_t)p.w_numel * p.elem();
    if (slice == 0 || slice > NOALLOC_SCRATCH_BYTES)
        return fail(OEQ_ERR_UNSUPPORTED, "weight tensor of " + std::to_string(slice) + " bytes exceeds the built-in scratch of " +
                                             std::to_string(NOALLOC_SCRATCH_BYTES) + " bytes; use oeq_tp_backward with caller scratch");
    const long long max_slices = (long long)(NOALLOC_SCRATCH_BYTES / slice);
    cudaStream_t st = (cudaStream_t)stream;
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    h->last_stream = st;       // oeq_tp_check synchronises the stream of the most recent launch
    if (p.mode == OEQ_MODE_UVW) {
        // always the FMA kernel: the tensor-core kernels want packed weight copies that only cudaMalloc gives
        if ((rc = load_uvw(h->bwd, p, true))) return rc;
        long long ctas = std::min(uvw_grid(h->bwd, batch), max_slices);
        UvwParams up{};
        up.X = X; up.Y = Y; up.W = W; up.dZ = dZ; up.dX = dX; up.dY = dY; up.dW = dW; up.ws = scratch;
        up.batch = batch; up.status = h->d_status;
        void* args[] = {&up};
        OEQ_CUDA(cudaLaunchKernel((const void*)h->bwd.fn, dim3((unsigned)ctas), dim3((unsigned)h->bwd.uvw.threads), args,
                                  (size_t)h->bwd.smem, st));
        int n = p.w_numel;
        const void* ws = scratch;
        void* rargs[] = {&ws, &dW, &n, &ctas};
        OEQ_CUDA(cudaLaunchKernel((const void*)h->bwd.reduce_fn, dim3((n + 31) / 32), dim3(256), rargs, 0, st));
        return OEQ_OK;
    }
    if ((rc = load_kernel(h->bwd, "oeq_uvu_kernel", true))) return rc;
    Kernel& k = h->bwd;
    const long long max_ctas = max_slices / k.map.ng;
    if (max_ctas < 1)
        return fail(OEQ_ERR_UNSUPPORTED, "one CTA's partial gradients exceed the built-in scratch; use oeq_tp_backward");
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.dZ = dZ; prm.dX = dX; prm.dY = dY; prm.dW = dW;
    prm.n_items = batch; prm.n_nodes = batch; prm.status = h->d_status; prm.ws = scratch;
    long long grid = 0;
    if ((rc = launch_uvu(k, p, prm, st, 0, max_ctas, &grid))) return rc;
    long long groups = grid * k.map.ng;
    int n = p.w_numel;
    const void* ws = scratch;
    void* rargs[] = {&ws, &dW, &n, &groups};
    OEQ_CUDA(cudaLaunchKernel((const void*)k.reduce_fn, dim3((n + 31) / 32), dim3(256), rargs, 0, st));
    return OEQ_OK;
}

// ---------------------------------------------------------------- fused convolution

int oeq_conv_create(const oeq_problem_desc* desc, int deterministic, oeq_conv** out) {
    if (!out) return fail(OEQ_ERR_INVALID, "null output handle");
    *out = nullptr;
    oeq_conv* h = new oeq_conv();
    h->deterministic = deterministic != 0;
    int rc = ingest(desc, h->prob);
    if (!rc) rc = check_conv_problem(h->prob);
    // what the problem's launches use: slice kernels where it has their shape (the group kernels behind them are then
    // only for lists beyond 32-bit counts, specialised on demand, and the receiver-order group kernel for wide rows)
    auto optional = [&](int rc2, bool& has) {
        has = rc2 == OEQ_OK;
        if (rc2 != OEQ_OK && rc2 != OEQ_ERR_UNSUPPORTED) rc = rc2;
    };
    if (!rc) optional(build_slice_fwd(h->prob, h->deterministic, h->fwd_slice), h->has_fwd_slice);
    if (!rc && (!h->has_fwd_slice || group_forward_beside_slice(h->prob, h->fwd_slice)))
        rc = build_uvu(h->prob, deterministic ? K_FWD_DET : K_FWD_ATOMIC, h->fwd);
    if (!rc) rc = build_uvu(h->prob, deterministic ? K_BWD_DET : K_BWD_ATOMIC, h->bwd);
    UvuTcGeometry geo;
    if (!rc && uvu_tc_geometry(h->prob, geo)) {
        rc = build_uvu_tc(h->prob, h->deterministic, h->fwd_tc);
        h->has_fwd_tc = !rc;
    }
    if (!rc) optional(build_slice_bwd(h->prob, h->deterministic, h->bwd_slice), h->has_bwd_slice);
    if (!rc && recv_beside_slice(h->prob, h->has_bwd_slice, h->bwd_slice, h->deterministic) && recv_backward_supported(h->prob)) {
        rc = build_uvu_recv(h->prob, h->deterministic, h->bwd_recv);
        h->has_bwd_recv = !rc;
    }
    if (rc) {
        delete h;
        return rc;
    }
    *out = h;
    return OEQ_OK;
}

int oeq_conv_destroy(oeq_conv* h) {
    if (!h) return OEQ_OK;
    if (h->d_status) cudaFree(h->d_status);
    if (h->fwd.lib) cudaLibraryUnload(h->fwd.lib);
    if (h->bwd.lib) cudaLibraryUnload(h->bwd.lib);
    if (h->fwd_tc.lib) cudaLibraryUnload(h->fwd_tc.lib);
    if (h->fwd_slice.lib) cudaLibraryUnload(h->fwd_slice.lib);
    if (h->bwd_slice.lib) cudaLibraryUnload(h->bwd_slice.lib);
    if (h->bwd_recv.lib) cudaLibraryUnload(h->bwd_recv.lib);
    if (h->dbl_z.lib) cudaLibraryUnload(h->dbl_z.lib);
    if (h->dbl_g.lib) cudaLibraryUnload(h->dbl_g.lib);
    delete h;
    return OEQ_OK;
}

// Scratch row of one edge in the deterministic receiver-order backward pass.
static size_t recv_row_bytes(const Problem& p) { return (size_t)pad16(p.x_dim * p.elem()); }
// Below this many scratch rows (when the edges do not all fit) the sender-order kernel is used instead.
static long long recv_min_block_edges() { return std::max(1, env_int("OEQ_B200_BWD_MIN_BLOCK", 1 << 16)); }

size_t oeq_conv_workspace_bytes(const oeq_conv* h, int64_t nodes, int64_t edges) {
    (void)nodes;
    // Forward: none (the segmented reduction is node-aligned: no scratch, no fix-up pass).  Deterministic
    // backward: one dX row per edge, capped (the pass then runs over blocks of edges); optional -- without
    // it the sender-order kernel runs.
    if (!h || !h->deterministic || !(h->has_bwd_recv || h->has_bwd_slice) || edges <= 0) return 0;
    const size_t cap = (size_t)std::max(1, env_int("OEQ_B200_BWD_SCRATCH_MB", 8192)) << 20;
    return std::min((size_t)edges * recv_row_bytes(h->prob), cap);
}

int oeq_conv_forward(oeq_conv* h, int64_t nodes, int64_t edges, const void* X, const void* Y, const void* W,
                     const int64_t* rows, const int64_t* cols, void* Z, void* workspace, size_t workspace_bytes,
                     void* stream) {
    (void)workspace; (void)workspace_bytes;
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (nodes < 0 || edges < 0) return fail(OEQ_ERR_INVALID, "negative size");
    cudaStream_t st = (cudaStream_t)stream;
    const Problem& p = h->prob;
    if (nodes == 0) return OEQ_OK;
    if (!Z) return fail(OEQ_ERR_INVALID, "null buffer");
    if (edges == 0 || !h->deterministic)
        OEQ_CUDA(cudaMemsetAsync(Z, 0, (size_t)nodes * p.z_dim * p.elem(), st));
    if (edges == 0) return OEQ_OK;
    if (!X || !Y || (!W && !p.unit) || !rows || !cols) return fail(OEQ_ERR_INVALID, "null buffer");
    // the tensor-core kernel stages rows with bulk copies only: it needs 16-byte aligned X and W
    const bool tc = h->has_fwd_tc && aligned16(X) && aligned16(W) && !env_int("OEQ_B200_NO_BULK", 0);
    int rc = ensure_status(&h->d_status);
    // (the slice kernels count nodes and edges in 32 bits)
    const bool group = h->has_fwd_slice && group_forward_beside_slice(p, h->fwd_slice) && (size_t)nodes * p.x_dim * p.elem() > GROUP_FORWARD_BYTES;
    if (!rc && !tc && h->has_fwd_slice && !group && edges < (1ll << 31) - 4096 && nodes < (1ll << 31) - 4096) {
        if ((rc = load_kernel(h->fwd_slice, "oeq_uvu_kernel", false))) return rc;
        UvuParams prm{};
        prm.X = X; prm.Y = Y; prm.W = W; prm.Z = Z;
        prm.rows = (const long long*)rows; prm.cols = (const long long*)cols;
        prm.n_items = edges; prm.n_nodes = nodes; prm.status = h->d_status;
        h->last_stream = st;
        return launch_slice(h->fwd_slice, p, prm, st);
    }
    if (!rc && !tc && !h->fwd.compiled) rc = build_uvu(p, h->deterministic ? K_FWD_DET : K_FWD_ATOMIC, h->fwd);
    if (!rc) rc = tc ? load_kernel(h->fwd_tc, "oeq_uvu_tc_kernel", false) : load_kernel(h->fwd, "oeq_uvu_kernel", false);
    if (rc) return rc;
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.Z = Z;
    prm.rows = (const long long*)rows; prm.cols = (const long long*)cols;
    prm.n_items = edges; prm.n_nodes = nodes; prm.status = h->d_status;
    h->last_stream = st;
#ifdef OEQ_DEV_PROFILE
    if (tc && env_int("OEQ_B200_TC_PROFILE", 0)) {
        // cycle accounting of the roles of CTA 0 (development aid): synchronous, prints to stderr
        unsigned long long* d = nullptr;
        OEQ_CUDA(cudaMalloc(&d, 64 * 8));
        OEQ_CUDA(cudaMemsetAsync(d, 0, 64 * 8, st));
        prm.ws = d;
        rc = launch_uvu(h->fwd_tc, p, prm, st);
        unsigned long long hbuf[64];
        OEQ_CUDA(cudaMemcpyAsync(hbuf, d, sizeof hbuf, cudaMemcpyDeviceToHost, st));
        OEQ_CUDA(cudaStreamSynchronize(st));
        cudaFree(d);
        const char* names[] = {"consumer0", "consumer1", "mma", "-", "stager"};
        for (int r = 0; r < 5; ++r)
            fprintf(stderr, "[oeq_b200 tc profile] %-9s total %llu  s1 %llu  s2 %llu  s3 %llu  s4 %llu  s5 %llu  s6 %llu  s7 %llu\n",
                    names[r], hbuf[8 * r], hbuf[8 * r + 1], hbuf[8 * r + 2], hbuf[8 * r + 3], hbuf[8 * r + 4], hbuf[8 * r + 5],
                    hbuf[8 * r + 6], hbuf[8 * r + 7]);
        return rc;
    }
#endif
    return launch_uvu(tc ? h->fwd_tc : h->fwd, p, prm, st);
}

int oeq_conv_backward(oeq_conv* h, int64_t nodes, int64_t edges, const void* X, const void* Y, const void* W,
                      const void* dZ, const int64_t* rows, const int64_t* cols, const int64_t* perm, void* dX,
                      void* dY, void* dW, void* workspace, size_t workspace_bytes, void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (nodes < 0 || edges < 0) return fail(OEQ_ERR_INVALID, "negative size");
    cudaStream_t st = (cudaStream_t)stream;
    const Problem& p = h->prob;
    if (nodes == 0) return OEQ_OK;
    if (!dX) return fail(OEQ_ERR_INVALID, "null buffer");
    if (edges == 0 || !h->deterministic)
        OEQ_CUDA(cudaMemsetAsync(dX, 0, (size_t)nodes * p.x_dim * p.elem(), st));
    if (edges == 0) return OEQ_OK;
    if (!X || !Y || !dZ || !rows || !cols || !dY || ((!W || !dW) && !p.unit))
        return fail(OEQ_ERR_INVALID, "null buffer");
    if (h->deterministic && !perm)
        return fail(OEQ_ERR_INVALID, "deterministic backward needs the sender-order permutation");
    int rc = ensure_status(&h->d_status);
    if (rc) return rc;
    h->last_stream = st;
    const int e = p.elem();
    // receiver-order pass: atomic variant always (dX was cleared above); deterministic variant when the
    // caller's scratch holds the rows of a useful block of edges
    const size_t row = recv_row_bytes(p);
    long long block_edges = 0;
    // (slice kernels count edges and nodes in 32 bits)
    const bool sliced = h->has_bwd_slice && edges < (1ll << 31) - 4096 && nodes < (1ll << 31) - 4096 &&
                        !(h->has_bwd_recv && edges >= recv_min_edges(h->deterministic));
    if (h->has_bwd_recv || sliced) {
        if (!h->deterministic) block_edges = edges;
        else if (workspace && aligned16(workspace)) {
            block_edges = (long long)std::min<size_t>(workspace_bytes / row, (size_t)edges);
            if (block_edges < edges && block_edges < recv_min_block_edges()) block_edges = 0;
        }
    }
    if (block_edges > 0) {
        Kernel& k = sliced ? h->bwd_slice : h->bwd_recv;
        if (!k.loaded) {
            if ((rc = load_kernel(k, "oeq_uvu_kernel", false))) return rc;
            if (h->deterministic) {
                OEQ_CUDA(cudaLibraryGetKernel(&h->sum_rows_fn, k.lib, "oeq_sum_sender_rows"));
                OEQ_CUDA(cudaLibraryGetKernel(&h->clear_fn, k.lib, "oeq_clear"));
            }
        }
        const char* Yb = (const char*)Y; const char* Wb = (const char*)W;
        char* dYb = (char*)dY; char* dWb = (char*)dW;
        h->last_bwd_launches = 0;
        const int dx_bulk = ((p.x_dim * e) % 16 == 0 && aligned16(dX)) ? 32 : 0;
        auto launch = [&](UvuParams& prm) { return sliced ? launch_slice(k, p, prm, st) : launch_uvu(k, p, prm, st, dx_bulk); };
        const int sum_chunk = row_sum_chunk(k, p, edges);
        auto pass1 = [&](long long e0, long long n, void* scratch, UvuParams& prm) {
            prm.X = X; prm.dZ = dZ; prm.dX = dX;
            prm.Y = Yb + (size_t)e0 * p.y_dim * e; prm.W = Wb + (size_t)e0 * p.w_numel * e;
            prm.dY = dYb + (size_t)e0 * p.y_dim * e; prm.dW = dWb + (size_t)e0 * p.w_numel * e;
            prm.rows = (const long long*)rows + e0; prm.cols = (const long long*)cols + e0;
            prm.n_items = n; prm.n_nodes = nodes; prm.status = h->d_status;
            prm.ws = scratch;
        };
        if (!h->deterministic) {
            UvuParams prm{};
            pass1(0, edges, nullptr, prm);
            if ((rc = launch(prm))) return rc;
            h->last_bwd_launches = 1;
            return OEQ_OK;
        }
        auto sum_launch = [&](long long e0, long long n, void* scratch, bool first) -> int {
            UvuParams sp{};
            sp.dX = dX; sp.ws = scratch;
            sp.rows = (const long long*)rows; sp.cols = (const long long*)cols; sp.perm = (const long long*)perm;
            sp.n_items = edges; sp.n_nodes = nodes; sp.status = h->d_status;
            sp.flags = (first ? 64 : 0) | (n == edges ? 128 : 0);
            sp.chunk = sum_chunk;
            sp.e_lo = e0; sp.e_hi = e0 + n;
            const long long grid = row_sum_grid(k, p, edges, sp.chunk);
            void* args[] = {&sp};
            OEQ_CUDA(cudaLaunchKernel((const void*)h->sum_rows_fn, dim3((unsigned)grid), dim3(256), args, 0, st));
            ++h->last_bwd_launches;
            return OEQ_OK;
        };
        // With helper warps the scratch is used as two halves: launch b writes the rows of block b into half
        // b % 2 while its helper warps sum block b - 1 from the other half; the last block is summed by a
        // launch of its own.  Blocks are kept above a minimum size, and a list that fits one half is still cut
        // into a few blocks so that most of the summing hides behind the receiver-order launches.
        // Pipelining pays when a block's receiver-order launch runs for a millisecond or more; the scratch
        // bytes of a block are a fair proxy for that (wide rows mean much arithmetic per edge).
        const size_t min_block_bytes = (size_t)std::max(1, env_int("OEQ_B200_PIPELINE_BLOCK_MB", 1024)) << 20;
        const long long min_block = std::max<long long>(recv_min_block_edges(), (long long)(min_block_bytes / row));
        const bool pipelined = k.map.helper_warps > 0 && edges >= 4 * min_block;
        // several blocks: rows of nodes that send nothing are never written by the row sum (cleared by a kernel: a
        // memset call may land on a copy engine behind the caller's host transfers)
        if (pipelined || block_edges < edges) {
            unsigned long long words = (unsigned long long)nodes * p.x_dim * e / 4;
            void* ptr = dX;
            void* args[] = {&ptr, &words};
            const unsigned grid = (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((unsigned long long)k.sm_count * 8, (words / 4 + 255) / 256));
            OEQ_CUDA(cudaLaunchKernel((const void*)h->clear_fn, dim3(grid), dim3(256), args, 0, st));
            ++h->last_bwd_launches;
        }
        if (pipelined) {
            const long long half = (long long)(workspace_bytes / row / 2);
            long long be = std::min<long long>(half, (edges + 3) / 4);
            be = std::max<long long>(be, std::min<long long>(half, min_block));
            if (be >= 1) {
                char* halves[2] = {(char*)workspace, (char*)workspace + (size_t)half * row};
                long long prev_e0 = -1, prev_n = 0;
                int b = 0;
                for (long long e0 = 0; e0 < edges; e0 += be, ++b) {
                    const long long n = std::min(be, edges - e0);
                    UvuParams prm{};
                    pass1(e0, n, halves[b & 1], prm);
                    if (prev_e0 >= 0) {
                        prm.sum_cols = (const long long*)cols; prm.sum_perm = (const long long*)perm;
                        prm.sum_ws = halves[(b - 1) & 1];
                        prm.sum_items = edges; prm.sum_e_lo = prev_e0; prm.sum_e_hi = prev_e0 + prev_n;
                        prm.sum_first = b == 1; prm.sum_chunk = sum_chunk;
                    }
                    if ((rc = launch(prm))) return rc;
                    ++h->last_bwd_launches;
                    prev_e0 = e0; prev_n = n;
                }
                return sum_launch(prev_e0, prev_n, halves[(b - 1) & 1], b == 1);
            }
        }
        bool first = true;
        for (long long e0 = 0; e0 < edges; e0 += block_edges) {
            const long long n = std::min(block_edges, edges - e0);
            UvuParams prm{};
            pass1(e0, n, workspace, prm);
            if ((rc = launch(prm))) return rc;
            ++h->last_bwd_launches;
            if ((rc = sum_launch(e0, n, workspace, first))) return rc;
            first = false;
        }
        return OEQ_OK;
    }
    if ((rc = load_kernel(h->bwd, "oeq_uvu_kernel", false))) return rc;
    h->last_bwd_launches = 1;
    UvuParams prm{};
    prm.X = X; prm.Y = Y; prm.W = W; prm.dZ = dZ; prm.dX = dX; prm.dY = dY; prm.dW = dW;
    prm.rows = (const long long*)rows; prm.cols = (const long long*)cols; prm.perm = (const long long*)perm;
    prm.n_items = edges; prm.n_nodes = nodes; prm.status = h->d_status;
#ifdef OEQ_DEV_PROFILE
    if (env_int("OEQ_B200_UVU_PROFILE", 0)) {
        // cycle accounting of CTA 0's first group (development aid): synchronous, prints to stderr
        unsigned long long* d = nullptr;
        OEQ_CUDA(cudaMalloc(&d, 8 * 8));
        OEQ_CUDA(cudaMemsetAsync(d, 0, 8 * 8, st));
        prm.ws = d;
        rc = launch_uvu(h->bwd, p, prm, st, 16);
        unsigned long long hb[8];
        OEQ_CUDA(cudaMemcpyAsync(hb, d, sizeof hb, cudaMemcpyDeviceToHost, st));
        OEQ_CUDA(cudaStreamSynchronize(st));
        cudaFree(d);
        fprintf(stderr, "[oeq_b200 conv backward profile] consumer: cycles %llu waiting for rows %llu items %llu | producer: cycles %llu "
                        "waiting for a stage %llu walking %llu issuing %llu\n", hb[0], hb[1], hb[2], hb[4], hb[5], hb[6], hb[7]);
        return rc;
    }
#endif
    return launch_uvu(h->bwd, p, prm, st);
}

// ---------------------------------------------------------------- second derivatives of the convolution

int oeq_conv_has_double_backward(const oeq_conv* h) {
    return h && h->dbl_state >= 0 && conv_second_possible(h->prob) ? 1 : 0;
}

int oeq_conv_double_backward(oeq_conv* h, int64_t nodes, int64_t edges, const void* X, const void* Y, const void* W,
                             const void* dZ, const void* EX, const void* EY, const void* EW, const int64_t* rows,
                             const int64_t* cols, const int64_t* perm, void* GX, void* GY, void* GW, void* GdZ,
                             void* workspace, size_t workspace_bytes, void* stream) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    std::lock_guard<std::mutex> lock(h->mutex);
    if (nodes < 0 || edges < 0) return fail(OEQ_ERR_INVALID, "negative size");
    if (!oeq_conv_has_double_backward(h)) return fail(OEQ_ERR_UNSUPPORTED, "no fused second derivatives for this problem");
    cudaStream_t st = (cudaStream_t)stream;
    const Problem& p = h->prob;
    if (nodes == 0) return OEQ_OK;
    if (!GX || !GdZ) return fail(OEQ_ERR_INVALID, "null buffer");
    const int e = p.elem();
    if (edges == 0) {
        OEQ_CUDA(cudaMemsetAsync(GX, 0, (size_t)nodes * p.x_dim * e, st));
        OEQ_CUDA(cudaMemsetAsync(GdZ, 0, (size_t)nodes * p.z_dim * e, st));
        return OEQ_OK;
    }
    if (!X || !Y || !W || !dZ || !EX || !EY || !EW || !rows || !cols || !GY || !GW) return fail(OEQ_ERR_INVALID, "null buffer");
    if (h->deterministic && !perm) return fail(OEQ_ERR_INVALID, "deterministic second derivatives need the sender-order permutation");
    const size_t row = recv_row_bytes(p);
    long long block_edges = edges;
    if (h->deterministic) {
        if (!workspace || !aligned16(workspace)) return fail(OEQ_ERR_UNSUPPORTED, "deterministic second derivatives need scratch memory");
        block_edges = (long long)std::min<size_t>(workspace_bytes / row, (size_t)edges);
        if (block_edges < edges && block_edges < recv_min_block_edges())
            return fail(OEQ_ERR_UNSUPPORTED, "deterministic second derivatives need more scratch memory");
    }
    int rc = ensure_status(&h->d_status);
    if (rc) return rc;
    if (h->dbl_state == 0) {
        rc = build_conv_dbl(p, h->deterministic, h->dbl_z, h->dbl_g);
        if (!rc) rc = load_kernel(h->dbl_z, "oeq_uvu_kernel", false);
        if (!rc) rc = load_kernel(h->dbl_g, "oeq_uvu_kernel", false);
        if (!rc) {
            OEQ_CUDA(cudaLibraryGetKernel(&h->dbl_sum_fn, h->dbl_g.lib, "oeq_sum_sender_rows"));
            OEQ_CUDA(cudaLibraryGetKernel(&h->dbl_clear_fn, h->dbl_g.lib, "oeq_clear"));
        }
        h->dbl_state = rc ? -1 : 1;
        if (rc) return rc;
    }
    const bool sliced = h->dbl_g.map.slice_warps > 0;
    if (sliced && (edges >= (1ll << 31) - 4096 || nodes >= (1ll << 31) - 4096))
        return fail(OEQ_ERR_UNSUPPORTED, "fused second derivatives count nodes and edges in 32 bits");
    h->last_stream = st;
    // bulk copies of a kind of row only when the row and its cotangent row both qualify
    int clear = 0;
    if (!aligned16(EX)) clear |= 1;
    if (!aligned16(EY)) clear |= 2;
    if (!aligned16(EW)) clear |= 4;
    // gradient with respect to dZ: the forward walk over all edges
    if (!h->deterministic) OEQ_CUDA(cudaMemsetAsync(GdZ, 0, (size_t)nodes * p.z_dim * e, st));
    {
        UvuParams prm{};
        prm.X = X; prm.Y = Y; prm.W = W; prm.Z = GdZ; prm.EX = EX; prm.EY = EY; prm.EW = EW;
        prm.rows = (const long long*)rows; prm.cols = (const long long*)cols;
        prm.n_items = edges; prm.n_nodes = nodes; prm.status = h->d_status;
        rc = sliced ? launch_slice(h->dbl_z, p, prm, st, clear) : launch_uvu(h->dbl_z, p, prm, st, 0, 0, nullptr, clear);
        if (rc) return rc;
    }
    // gradients with respect to X, Y, W: the receiver-order walk, GX through scratch rows or bulk reductions
    Kernel& k = h->dbl_g;
    if (!h->deterministic || block_edges < edges) {     // (one row sum over the whole list writes every row itself)
        unsigned long long words = (unsigned long long)nodes * p.x_dim * e / 4;
        void* ptr = GX;
        void* args[] = {&ptr, &words};
        const unsigned grid = (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((unsigned long long)k.sm_count * 8, (words / 4 + 255) / 256));
        OEQ_CUDA(cudaLaunchKernel((const void*)h->dbl_clear_fn, dim3(grid), dim3(256), args, 0, st));
    }
    const int dx_bulk = ((p.x_dim * e) % 16 == 0 && aligned16(GX)) ? 32 : 0;
    const int sum_chunk = row_sum_chunk(k, p, edges);
    bool first = true;
    for (long long e0 = 0; e0 < edges; e0 += block_edges) {
        const long long n = std::min(block_edges, edges - e0);
        const size_t yo = (size_t)e0 * p.y_dim * e, wo = (size_t)e0 * p.w_numel * e;
        UvuParams prm{};
        prm.X = X; prm.dZ = dZ; prm.dX = GX; prm.EX = EX;
        prm.Y = (const char*)Y + yo; prm.W = (const char*)W + wo;
        prm.EY = (const char*)EY + yo; prm.EW = (const char*)EW + wo;
        prm.dY = (char*)GY + yo; prm.dW = (char*)GW + wo;
        prm.rows = (const long long*)rows + e0; prm.cols = (const long long*)cols + e0;
        prm.n_items = n; prm.n_nodes = nodes; prm.status = h->d_status;
        prm.ws = h->deterministic ? workspace : nullptr;
        rc = sliced ? launch_slice(k, p, prm, st, clear) : launch_uvu(k, p, prm, st, dx_bulk, 0, nullptr, clear);
        if (rc) return rc;
        if (h->deterministic) {
            UvuParams sp{};
            sp.dX = GX; sp.ws = workspace;
            sp.rows = (const long long*)rows; sp.cols = (const long long*)cols; sp.perm = (const long long*)perm;
            sp.n_items = edges; sp.n_nodes = nodes; sp.status = h->d_status;
            sp.flags = (first ? 64 : 0) | (n == edges ? 128 : 0);
            sp.chunk = sum_chunk;
            sp.e_lo = e0; sp.e_hi = e0 + n;
            const long long grid = row_sum_grid(k, p, edges, sp.chunk);
            void* args[] = {&sp};
            OEQ_CUDA(cudaLaunchKernel((const void*)h->dbl_sum_fn, dim3((unsigned)grid), dim3(256), args, 0, st));
            first = false;
        }
    }
    return OEQ_OK;
}

// ---------------------------------------------------------------- self-test of the bounded waits

// One thread waits on a shared-memory barrier that nothing ever completes, polls `polls` times, gives up, records
// the code in *status and returns: the path every staged kernel takes when a copy never lands.
__global__ void oeq_wait_probe_kernel(int* status, unsigned polls) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0) {
        oeq::mbar_init(&bar, 1);
        oeq::fence_mbar_init();
        bool done = false;
        for (unsigned spin = 0; spin < polls && !done; ++spin) done = oeq::mbar_try_wait(&bar, 0u);
        if (!done) atomicCAS(status, 0, oeq::ERR_WAIT_FULL);
    }
}

int oeq_selftest_bounded_wait(int polls, void* stream) {
    if (polls < 1 || polls > (1 << 20)) return fail(OEQ_ERR_INVALID, "polls must be in 1 .. 2^20");
    int* d_status = nullptr;
    int rc = ensure_status(&d_status);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    oeq_wait_probe_kernel<<<1, 32, 0, st>>>(d_status, (unsigned)polls);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) rc = check_status(d_status, st);      // OEQ_ERR_DEVICE_WAIT is the expected answer
    cudaFree(d_status);
    if (e != cudaSuccess) return fail(OEQ_ERR_CUDA, std::string("wait probe: ") + cudaGetErrorString(e));
    return rc;
}

int oeq_conv_last_backward_launches(const oeq_conv* h) { return h ? h->last_bwd_launches : 0; }

int oeq_conv_check(oeq_conv* h) { return h ? check_status(h->d_status, h->last_stream) : fail(OEQ_ERR_INVALID, "null handle"); }

int oeq_conv_launch_info(const oeq_conv* h, int which, int* threads, int* ng, int* ps, int* stages, int* smem, int* regs) {
    if (!h) return fail(OEQ_ERR_INVALID, "null handle");
    const Kernel& k = which ? (h->bwd_slice.loaded ? h->bwd_slice : h->bwd_recv.loaded ? h->bwd_recv : h->bwd)
                            : (h->fwd_tc.loaded ? h->fwd_tc : h->has_fwd_slice ? h->fwd_slice : h->fwd);
    return launch_info(k, threads, ng, ps, stages, smem, regs);
}

}  // extern "C"
