// ensemble.cu -- independent QGN members with different grid sizes and layer counts,
// advanced together with BSRK3 (BSRK3.f90) in FP64 or in the mixed mode.
//
// Every pass of an attempt -- stage combination + GetPsi, the three right-hand-side passes,
// the error combination, the error transform and the controller -- is ONE launch for the
// whole ensemble (the x pass: one per grid size): a table maps each CTA, or each turn of a
// persistent grid-stride loop, to a member and a tile, and the tile bodies of the single-field kernels (rhs_tiles.cuh) run
// on it with the member's geometry.  All members take their attempts in lockstep; members
// that have taken their steps (or halted) drop out of the tile loops.  The attempts of an
// advance run as the body of a CUDA graph WHILE node whose condition the controller kernel
// sets on the device ("any member still active"), so an advance is one graph launch.  An
// autotuner times each pass's tile-width variants and grid sizes on the ensemble at hand
// the first time it advances and keeps the fastest.
//
// Members are ordinary contexts (qgn_create, scheme BSRK3) that the ensemble borrows: their
// buffers, constants and device scalars are used in place, so qgn_get_state, qgn_rhs,
// qgn_physical and the diagnostics keep working on each member.  In the mixed mode the
// stage right-hand sides, stage inputs and psi are FP32 and the transforms run in FP32; the
// state, the stage sums (accumulated in FP64), GetPsi's arithmetic, the error combination,
// its transform and the controller are FP64.
#include "qgn_internal.cuh"
#include "fft.cuh"
#include "prof.cuh"
#include "rhs_tiles.cuh"
#include "ctrl.cuh"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <string>
#include <unordered_set>
#include <vector>

namespace qgn {
namespace {

// one row of the device member table
struct EnsMember {
    Geom g;
    double2* q;           // accepted state (FP64)
    double2* qc;          // fourth-stage state q_tmp, the candidate solution (FP64)
    double2* err;         // embedded error spectrum (FP64)
    void* N[4];           // RHS0..RHS3 in the stage precision
    void* Qs;             // stage input in the stage precision
    void* psi;            // GetPsi of the stage input
    void* hq;             // half-transformed fields (stage precision; FP64 for the error transform)
    void* hp;
    void* hu;
    void* hpp;
    void* hpd;
    const void* twx;      // twiddles in the stage precision
    const void* twy;
    const double2* twx64;
    const double2* twy64;
    const LayerConst* lc;
    const ModalConst* mc;
    DevScalars* sc;
    double TOL, dt_max;
    int max_rejects;
    int steps_left;       // accepted steps still to take in this advance
    int active;           // 1 while steps_left > 0 and the member has not halted
    int need_fsal;        // RHS0 of the current state is still to be computed
};

// passes with their own tile tables (EP_XPASS: one per grid size)
enum { EP_POINT = 0, EP_ELEM, EP_YINV, EP_XPASS, EP_YFWD, EP_YINV1, EP_XINV1, EP_COUNT };
// passes the autotuner chooses for
enum { TP_YINV = 0, TP_XPASS, TP_YFWD, TP_COUNT };
// Tile variants the autotuner searches per pass: CTA width (threads of a y pass, threads per
// slot group of the x pass) and elements per thread of the transforms (tv_make, rhs_tiles.cuh).
// Every listed pair gives whole tiles for 128-, 256- and 512-point transforms (the y-forward
// needs a width of at least two transforms, the others one); 32 elements per thread only in
// FP32, where they take 64 registers (FP64 would spill under the 128-register cap).  Index 1 is
// the default before tuning (16 elements per thread).
template <class CT>
struct EnsVariants;
template <>
struct EnsVariants<double2> {
    static constexpr int yinv[] = {tv_make(64, 16), tv_make(128, 16), tv_make(256, 16),
                                   tv_make(64, 8),  tv_make(128, 8),  tv_make(256, 8)};
    static constexpr int xpass[] = {tv_make(32, 16), tv_make(64, 16), tv_make(128, 16), tv_make(64, 8),
                                    tv_make(128, 8)};
    static constexpr int yfwd[] = {tv_make(64, 16), tv_make(128, 16), tv_make(256, 16), tv_make(128, 8),
                                   tv_make(256, 8)};
};
template <>
struct EnsVariants<float2> {
    static constexpr int yinv[] = {tv_make(64, 16), tv_make(128, 16), tv_make(256, 16), tv_make(64, 8),
                                   tv_make(128, 8),  tv_make(256, 8),  tv_make(64, 32),  tv_make(128, 32),
                                   tv_make(256, 32)};
    static constexpr int xpass[] = {tv_make(32, 16), tv_make(64, 16), tv_make(128, 16), tv_make(64, 8),
                                    tv_make(128, 8), tv_make(32, 32), tv_make(64, 32),  tv_make(128, 32)};
    static constexpr int yfwd[] = {tv_make(64, 16), tv_make(128, 16), tv_make(256, 16), tv_make(128, 8),
                                   tv_make(256, 8), tv_make(64, 32),  tv_make(128, 32)};
};
template <class CT>
constexpr int ens_variant_count(int tp) {
    return tp == 0 ? (int)(sizeof(EnsVariants<CT>::yinv) / sizeof(int))
                   : tp == 1 ? (int)(sizeof(EnsVariants<CT>::xpass) / sizeof(int))
                             : (int)(sizeof(EnsVariants<CT>::yfwd) / sizeof(int));
}
template <class CT>
constexpr int ens_variant(int tp, int v) {
    return tp == 0 ? EnsVariants<CT>::yinv[v] : tp == 1 ? EnsVariants<CT>::xpass[v] : EnsVariants<CT>::yfwd[v];
}
constexpr int kDefaultVariant = 1;
// register cap of an ensemble transform kernel: 32 FP32 elements per thread need 64 for data
template <class CT, int TV>
__host__ __device__ constexpr int ens_regcap() {
    return tv_radix(TV) == 32 ? 128 : regcap<CT>(128, 96);
}
constexpr int kPointTile = 256;

// The tiles of a pass: tile t is tile t - start[i] of entry i = map[t] (a member, or a member of a
// group).  Looked up, not searched for: five dependent loads before a CTA knew its member were a good
// part of the short kernels.
struct TileTab {
    const int* start;
    const int* map;
    int total;
};

// stage 0 is the FSAL evaluation RHS0 = GetRHS(q_hat) (BSRK3.f90:12-17), stages 1..3 the
// attempt's stages; a member takes part in a pass when it needs that evaluation
__device__ __forceinline__ bool ens_runs(const EnsMember& M, int stage) {
    return stage == 0 ? (M.need_fsal != 0 && M.active != 0) : M.active != 0;
}

template <class CT>
__device__ __forceinline__ CT to_ct(double2 v);
template <>
__device__ __forceinline__ double2 to_ct<double2>(double2 v) { return v; }
template <>
__device__ __forceinline__ float2 to_ct<float2>(double2 v) { return make_float2((float)v.x, (float)v.y); }

template <class CT>
__device__ __forceinline__ void axpy(double2& v, double c, CT r) {
    v.x += c * (double)r.x;
    v.y += c * (double)r.y;
}

// the field the stage-s right-hand side reads: FP64 stage 3 reads q_tmp in place
template <class CT>
__device__ __forceinline__ const CT* stage_input(const EnsMember& M, int s) {
    return (sizeof(CT) == 16 && s == 3) ? reinterpret_cast<const CT*>(M.qc) : static_cast<const CT*>(M.Qs);
}

// ---- stage combination + GetPsi (BSRK3.f90:21-28, QGN_Module.f90:315-341) ------------------
// One mode, all layers per thread.  The state and right-hand sides are requested before the mode
// matrices are staged, so that the tile's two dependent rounds of loads overlap; a noinline body
// per layer count, called after the staging, read them one round later: 32 members of 128^2 to 512^2
// took 106 us (FP32), now 72 us.  Latency-bound still: 16 warps per SM at 128 registers.
struct EnsModes {
    double proj[kMaxNZ * kMaxNZ], back[kMaxNZ * kMaxNZ], ev[kMaxNZ];
};

template <int NZ, class CT>
__device__ __forceinline__ void ens_stage_tile(const EnsMember& M, const Geom& g, int tile, int s, EnsModes& sm) {
    const unsigned P = (unsigned)(g.nkx * g.nky);
    const unsigned p = (unsigned)tile * kPointTile + threadIdx.x;
    const bool ok = p < P;
    double2 qv[NZ], pv[NZ];
    if (ok) {
        const double dt = M.sc->dt;
        const double2* q = M.q;
#pragma unroll
        for (int l = 0; l < NZ; ++l) qv[l] = q[(size_t)l * P + p];
        auto coef = [&](int j) {
            return (s == 1 ? 0.5 : s == 2 ? 0.75 : j == 0 ? 2.0 / 9.0 : j == 1 ? 1.0 / 3.0 : 4.0 / 9.0) * dt;
        };
        const int first = s == 2 ? 1 : 0, last = s == 3 ? 2 : s - 1;
        if (sizeof(CT) == 8 && s == 3) {   // FP32: all three right-hand sides requested at once
            CT r[3][NZ];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int l = 0; l < NZ; ++l) r[j][l] = (static_cast<const CT*>(M.N[j]) + p)[(size_t)l * P];
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int l = 0; l < NZ; ++l) axpy(qv[l], coef(j), r[j][l]);
        } else {
#pragma unroll 1
            for (int j = first; j <= last; ++j) {   // FP64: one right-hand side's layers at a time
                const double c = coef(j);
                const CT* R = static_cast<const CT*>(M.N[j]) + p;
                CT r[NZ];
#pragma unroll
                for (int l = 0; l < NZ; ++l) r[l] = R[(size_t)l * P];
#pragma unroll
                for (int l = 0; l < NZ; ++l) axpy(qv[l], c, r[l]);
            }
        }
    }
    for (int i = threadIdx.x; i < NZ * NZ; i += kPointTile) {
        sm.proj[i] = M.mc->proj[i];
        sm.back[i] = M.mc->back[i];
    }
    if (threadIdx.x < NZ) sm.ev[threadIdx.x] = M.mc->evals[threadIdx.x];
    __syncthreads();
    if (!ok) return;
    const int kx = (int)(p / (unsigned)g.nky), m = (int)(p % (unsigned)g.nky);
    const double kxv = g.dkx * kx, kyv = g.kyval(g.jfull(m));
    const double k2 = kxv * kxv + kyv * kyv;
    modal_invert<NZ>(sm.proj, sm.back, sm.ev, M.mc->Htot, NZ, k2, p == 0, qv, pv);
    CT* Qs = const_cast<CT*>(stage_input<CT>(M, s));
    CT* psi = static_cast<CT*>(M.psi);
    const bool keep = sizeof(CT) == 8 && s == 3;   // the FP64 candidate of the mixed mode
#pragma unroll
    for (int l = 0; l < NZ; ++l) {
        const size_t idx = (size_t)l * P + p;
        Qs[idx] = to_ct<CT>(qv[l]);
        psi[idx] = to_ct<CT>(pv[l]);
        if (keep) M.qc[idx] = qv[l];
    }
}

// one CTA per tile (in a loop over tiles every form of this spilled kilobytes per thread); NZ16: some
// member has 16 layers
template <class CT, bool NZ16>
__global__ void __launch_bounds__(kPointTile, 2)
    k_ens_stage(const EnsMember* __restrict__ mem, TileTab tab, int s) {
    QGN_PDL_ENTRY();
    __shared__ EnsModes sm;
    const int t = blockIdx.x;
    const int mi = tab.map[t];
    const EnsMember& M = mem[mi];
    if (!ens_runs(M, s)) return;
    const Geom g = M.g;
    const int tile = t - tab.start[mi];
    switch (g.nz) {
        case 2: ens_stage_tile<2, CT>(M, g, tile, s, sm); break;
        case 3: ens_stage_tile<3, CT>(M, g, tile, s, sm); break;
        case 4: ens_stage_tile<4, CT>(M, g, tile, s, sm); break;
        case 5: ens_stage_tile<5, CT>(M, g, tile, s, sm); break;
        case 6: ens_stage_tile<6, CT>(M, g, tile, s, sm); break;
        case 7: ens_stage_tile<7, CT>(M, g, tile, s, sm); break;
        case 8: ens_stage_tile<8, CT>(M, g, tile, s, sm); break;
        case 16:
            if constexpr (NZ16) ens_stage_tile<16, CT>(M, g, tile, s, sm);
            break;
        default: break;   // qgn_ens_create admits these layer counts only
    }
}

// ---- right-hand-side passes over all members ------------------------------------------------
template <int N, class CT, int TV>
__device__ __noinline__ void ens_yinv_one(const EnsMember& M, const Geom& g, int local, int s) {
    using C = YInvCfg<N, CT, TV>;
    static_assert(C::THREADS == tv_width(TV), "y-inverse tile width must give TV threads");
    const int nbx = (g.nkx + C::TKX - 1) / C::TKX;
    yinv_tile<N, 3, CT, TV>(g, threadIdx.x, local % nbx, local / nbx, stage_input<CT>(M, s), static_cast<const CT*>(M.psi),
                            static_cast<CT*>(M.hq), static_cast<CT*>(M.hp), static_cast<CT*>(M.hu),
                            static_cast<const CT*>(M.twy));
}

template <class CT, int TV>
__global__ void __launch_bounds__(tv_width(TV), minb(tv_width(TV), ens_regcap<CT, TV>()))
    k_ens_yinv(const EnsMember* __restrict__ mem, TileTab tab, int s) {
    QGN_PDL_ENTRY();
    for (int t = blockIdx.x; t < tab.total; t += gridDim.x) {
        const int mi = tab.map[t];
        const EnsMember& M = mem[mi];
        if (!ens_runs(M, s)) continue;
        const Geom g = M.g;
        const int local = t - tab.start[mi];
        switch (g.ny) {
            case 128: ens_yinv_one<128, CT, TV>(M, g, local, s); break;
            case 256: ens_yinv_one<256, CT, TV>(M, g, local, s); break;
            case 512: ens_yinv_one<512, CT, TV>(M, g, local, s); break;
            default: break;
        }
        __syncthreads();   // shared memory is reused by the next tile
    }
}

// The x pass of the members of one grid size (idx: their numbers).  The
// geometry is a kernel parameter, the row length a constant, and a CTA takes one tile: in a loop over
// tiles, the same body spills 0.4 to 0.8 KB per thread (in FP32 as well, at 96 registers), whether it
// is inlined or called, and in a call it also saves its registers on entry.  32 members of 128^2 to
// 512^2, FP32: one looping launch for all sizes 181 us, the three launches 112 us.
template <int N, class CT, int TV>
__global__ void __launch_bounds__(3 * tv_width(TV), minb(3 * tv_width(TV), ens_regcap<CT, TV>()))
    k_ens_xpass(Geom g, const EnsMember* __restrict__ mem, const int* __restrict__ idx, TileTab tab, int s) {
    QGN_PDL_ENTRY();
    using C = XCfg<N, false, CT, TV>;
    static_assert(C::THREADS == 3 * tv_width(TV), "x-pass tile width must give 3 TV threads");
    const int nbx = (g.ny / 2 + C::RP - 1) / C::RP;
    const int t = blockIdx.x;
    const int gi = tab.map[t];
    const EnsMember& M = mem[idx[gi]];
    if (!ens_runs(M, s)) return;
    const int local = t - tab.start[gi];
#ifdef QGN_CHECK
    Geom gm = M.g;     // this member's layer count bounds the checked indices
#else
    const Geom& gm = g;
#endif
    xpass_tile<N, false, CT, TV>(gm, threadIdx.x, local % nbx, local / nbx, static_cast<const CT*>(M.hq),
                                 static_cast<const CT*>(M.hp), static_cast<const CT*>(M.hu), static_cast<CT*>(M.hpp),
                                 static_cast<CT*>(M.hpd), static_cast<const CT*>(M.twx));
}

template <int N, class CT, int TV>
__device__ __noinline__ void ens_yfwd_one(const EnsMember& M, const Geom& g, int local, int s) {
    using C = YFwdCfg<N, false, CT, TV>;
    static_assert(C::THREADS == tv_width(TV), "y-forward tile width must give TV threads");
    const int nbx = (g.nkx + C::TKX - 1) / C::TKX;
    yfwd_tile<N, false, CT, TV>(g, threadIdx.x, local % nbx, local / nbx, M.lc, stage_input<CT>(M, s),
                                static_cast<const CT*>(M.psi), static_cast<const CT*>(M.hpp),
                                static_cast<const CT*>(M.hpd), static_cast<CT*>(M.N[s]),
                                static_cast<const CT*>(M.twy));
}

template <class CT, int TV>
__global__ void __launch_bounds__(tv_width(TV), minb(tv_width(TV), ens_regcap<CT, TV>()))
    k_ens_yfwd(const EnsMember* __restrict__ mem, TileTab tab, int s) {
    QGN_PDL_ENTRY();
    for (int t = blockIdx.x; t < tab.total; t += gridDim.x) {
        const int mi = tab.map[t];
        const EnsMember& M = mem[mi];
        if (!ens_runs(M, s)) continue;
        const Geom g = M.g;
        const int local = t - tab.start[mi];
        switch (g.ny) {
            case 128: ens_yfwd_one<128, CT, TV>(M, g, local, s); break;
            case 256: ens_yfwd_one<256, CT, TV>(M, g, local, s); break;
            case 512: ens_yfwd_one<512, CT, TV>(M, g, local, s); break;
            default: break;
        }
        __syncthreads();
    }
}

// ---- embedded error (BSRK3.f90:30-34), FP64 -------------------------------------------------
template <class CT>
__global__ void __launch_bounds__(256) k_ens_err(EnsMember* __restrict__ mem, TileTab tab) {
    QGN_PDL_ENTRY();
    for (int t = blockIdx.x; t < tab.total; t += gridDim.x) {
        const int mi = tab.map[t];
        const EnsMember& M = mem[mi];
        if (!M.active) continue;
        const int local = t - tab.start[mi];
        if (local == 0 && threadIdx.x == 0) {
            M.sc->maxbits = 0ULL;
            M.sc->accept = 0;
        }
        const size_t e = (size_t)local * kPointTile + threadIdx.x;
        if (e >= M.g.csize()) continue;
        double2 v = make_double2(0.0, 0.0);
        axpy(v, 5.0 / 72.0, static_cast<const CT*>(M.N[0])[e]);
        axpy(v, -1.0 / 12.0, static_cast<const CT*>(M.N[1])[e]);
        axpy(v, -1.0 / 9.0, static_cast<const CT*>(M.N[2])[e]);
        axpy(v, 1.0 / 8.0, static_cast<const CT*>(M.N[3])[e]);
        M.err[e] = v;
    }
}

// FP64 y-inverse of the error spectrum, then the x c2r with max|.| (err_phys, BSRK3.f90:35-37)
template <int N>
__device__ __noinline__ void ens_yinv1_one(const EnsMember& M, const Geom& g, int local) {
    using C = YInvCfg<N, double2, 128>;
    static_assert(C::THREADS == 128, "");
    const int nbx = (g.nkx + C::TKX - 1) / C::TKX;
    yinv_tile<N, 1, double2, 128>(g, threadIdx.x, local % nbx, local / nbx, M.err, nullptr, static_cast<double2*>(M.hq), nullptr,
                                  nullptr, M.twy64);
}

__global__ void __launch_bounds__(128, minb(128)) k_ens_yinv1(const EnsMember* __restrict__ mem,
                                                              TileTab tab) {
    QGN_PDL_ENTRY();
    for (int t = blockIdx.x; t < tab.total; t += gridDim.x) {
        const int mi = tab.map[t];
        const EnsMember& M = mem[mi];
        if (!M.active) continue;
        const Geom g = M.g;
        const int local = t - tab.start[mi];
        switch (g.ny) {
            case 128: ens_yinv1_one<128>(M, g, local); break;
            case 256: ens_yinv1_one<256>(M, g, local); break;
            case 512: ens_yinv1_one<512>(M, g, local); break;
            default: break;
        }
        __syncthreads();
    }
}

template <int N>
__device__ __noinline__ void ens_xinv1_one(const EnsMember& M, const Geom& g, int local) {
    using C = X1Cfg<N, 128>;
    static_assert(C::THREADS == 128, "");
    const int nbx = (g.ny / 2 + C::RP - 1) / C::RP;
    xinv1_tile<N, 0, 128>(g, local % nbx, local / nbx, static_cast<const double2*>(M.hq), M.sc, nullptr, M.twx64);
}

__global__ void __launch_bounds__(128, minb(128)) k_ens_xinv1(const EnsMember* __restrict__ mem,
                                                              TileTab tab) {
    QGN_PDL_ENTRY();
    for (int t = blockIdx.x; t < tab.total; t += gridDim.x) {
        const int mi = tab.map[t];
        const EnsMember& M = mem[mi];
        if (!M.active) continue;
        const Geom g = M.g;
        const int local = t - tab.start[mi];
        switch (g.nx) {
            case 128: ens_xinv1_one<128>(M, g, local); break;
            case 256: ens_xinv1_one<256>(M, g, local); break;
            case 512: ens_xinv1_one<512>(M, g, local); break;
            default: break;
        }
        __syncthreads();
    }
}

// ---- controller, arming and FSAL bookkeeping ------------------------------------------------
// BSRK3's accept/reject and PI update per member (BSRK3.f90:38-48); an accepted member
// takes q_tmp as its state and RHS3 as RHS0 by swapping table pointers.  The WHILE
// condition of the graph (and *any) says whether a member is still active.
__global__ void __launch_bounds__(256) k_ens_ctrl(EnsMember* __restrict__ mem, int nm,
                                                  cudaGraphConditionalHandle loop, int has_loop, int* __restrict__ any) {
    QGN_PDL_ENTRY();
    int act = 0;
    for (int i = threadIdx.x; i < nm; i += blockDim.x) {
        EnsMember& M = mem[i];
        if (M.active) {
            DevScalars* sc = M.sc;
            ctrl_decide(2, M.g.inv_nxny, M.TOL, M.dt_max, M.max_rejects, sc);
            if (sc->halt) {
                M.active = 0;
            } else if (sc->accept) {
                double2* tq = M.q;
                M.q = M.qc;
                M.qc = tq;
                void* tn = M.N[0];
                M.N[0] = M.N[3];
                M.N[3] = tn;
                sc->rejects_step = 0;
                if (--M.steps_left <= 0) M.active = 0;
            }
        }
        act |= M.active;
    }
    act = __syncthreads_or(act);
    if (threadIdx.x == 0) {
        *any = act;
        if (has_loop) cudaGraphSetConditional(loop, act ? 1u : 0u);
    }
}

__global__ void k_ens_arm(EnsMember* __restrict__ mem, int nm, int nsteps) {
    QGN_PDL_ENTRY();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nm; i += gridDim.x * blockDim.x) {
        EnsMember& M = mem[i];
        const bool go = nsteps > 0 && M.sc->halt == 0;
        M.steps_left = nsteps;
        M.active = go ? 1 : 0;
        if (go) M.sc->rejects_step = 0;
    }
}

__global__ void k_ens_fsal_done(EnsMember* __restrict__ mem, int nm) {
    QGN_PDL_ENTRY();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nm; i += gridDim.x * blockDim.x)
        if (mem[i].active) mem[i].need_fsal = 0;
}

// ---- host side --------------------------------------------------------------------------------
// opt a kernel into more than 48 KB of dynamic shared memory once per process, so that no
// attribute call happens while a graph is being captured
template <class K>
cudaError_t smem_attr(K kernel, int bytes) {
    return smem_opt_in(kernel, bytes);
}

template <class CT, int TV>
constexpr int yinv_smem() {
    return cmax(YInvCfg<128, CT, TV>::SMEM, cmax(YInvCfg<256, CT, TV>::SMEM, YInvCfg<512, CT, TV>::SMEM));
}
template <class CT, int TV>
constexpr int yfwd_smem() {
    return cmax(YFwdCfg<128, false, CT, TV>::SMEM,
                cmax(YFwdCfg<256, false, CT, TV>::SMEM, YFwdCfg<512, false, CT, TV>::SMEM));
}
constexpr int yinv1_smem() {
    return cmax(YInvCfg<128, double2, 128>::SMEM,
                cmax(YInvCfg<256, double2, 128>::SMEM, YInvCfg<512, double2, 128>::SMEM));
}
constexpr int xinv1_smem() {
    return cmax(X1Cfg<128, 128>::SMEM, cmax(X1Cfg<256, 128>::SMEM, X1Cfg<512, 128>::SMEM));
}

int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// threads per transform of n points at t elements per thread (FFTShape)
int fft_threads(int n, int t) { return n / std::min(n, t); }

// tiles of one member for a pass and tile variant (the tile shapes of YInvCfg, XCfg, YFwdCfg)
int member_tiles(const Geom& g, int pass, int tv) {
    const int w = tv_width(tv), r = tv_radix(tv) ? tv_radix(tv) : 16;
    const int Gx = fft_threads(g.nx, r), Gy = fft_threads(g.ny, r);
    const int G1x = g.nx / 16, G1y = g.ny / 16;   // the error transforms: 16 elements per thread
    switch (pass) {
        case EP_POINT: return ceil_div((long long)g.nkx * g.nky, kPointTile);
        case EP_ELEM: return ceil_div((long long)g.csize(), kPointTile);
        case EP_YINV: return ceil_div(g.nkx, std::max(1, w / Gy)) * g.nz;
        case EP_XPASS: return ceil_div(g.ny / 2, std::max(1, w / Gx)) * g.nz;
        case EP_YFWD: return ceil_div(g.nkx, std::min(std::max(1, w / (2 * Gy)), 16)) * g.nz;
        case EP_YINV1: return ceil_div(g.nkx, 128 / G1y) * g.nz;
        case EP_XINV1: return ceil_div(g.ny / 2, 128 / G1x) * g.nz;
        default: return 0;
    }
}

}  // namespace
}  // namespace qgn

using namespace qgn;

struct qgn_ens {
    std::vector<qgn_ctx*> mem;
    std::vector<long long> seen_version;
    int precision = QGN_PREC_FP64;
    int device = 0;
    cudaStream_t stream = nullptr;
    EnsMember* d_mem = nullptr;
    std::vector<EnsMember> h_mem;
    int* d_start = nullptr;          // EP_COUNT tables of nm+1 prefix sums
    std::vector<int> h_start;
    std::vector<int> h_map;          // tile -> member of every pass, the pass's part at map_at[pass]
    int map_at[EP_COUNT] = {};
    int* d_map = nullptr;
    size_t map_cap = 0;              // entries of d_map
    bool tables_new = true;          // built since the last upload
    int uploads = 0;
    // members of one grid size, for the x pass: their numbers and tile prefix sums at `table` of d_xgroups
    struct XGroup {
        int nx, ny;
        std::vector<int> members;
        int table = 0, tiles = 0, map_at = 0;
    };
    std::vector<XGroup> xgroups;
    std::vector<int> h_xgroups;      // per group: members, then their count + 1 prefix sums (tile -> member of
                                     // the group: h_map at map_at)
    int* d_xgroups = nullptr;
    int* d_any = nullptr;
    int* h_any = nullptr;            // pinned
    int variant[TP_COUNT] = {kDefaultVariant, kDefaultVariant, kDefaultVariant};
    // 0: one CTA per tile; k > 0: k CTAs per SM, persistent (y passes), or one CTA per tile and at most
    // k resident on an SM (x pass)
    int grid_mode[TP_COUNT] = {0, 0, 0};
    int smem_sm = 0, smem_cta = 0, smem_reserved = 0;   // shared memory: of an SM, most of a CTA, reserved per CTA
    float tuned_ms[TP_COUNT] = {0.f, 0.f, 0.f};
    bool pinned[TP_COUNT] = {false, false, false};   // set by qgn_ens_set_tiles: not tuned
    bool tuned = false;
    bool graphs_off = false;
    cudaGraphExec_t gexec = nullptr;
    long long g_body[KID_COUNT] = {};
    long long g_root[KID_COUNT] = {};
    Prof prof;
    std::string last_error;
    int sms = 148;
};

namespace {

struct EnsProfScope {
    Prof* prev;
    explicit EnsProfScope(qgn_ens* e) : prev(current_prof()) { current_prof() = &e->prof; }
    ~EnsProfScope() { current_prof() = prev; }
};

int ens_err(qgn_ens* e, int code, const std::string& msg) {
    e->last_error = msg;
    return code;
}

#define ECK(call)                                                                                   \
    do {                                                                                            \
        cudaError_t _e = (call);                                                                    \
        if (_e != cudaSuccess) {                                                                    \
            char _b[512];                                                                           \
            std::snprintf(_b, sizeof(_b), "%s: %s (%s)", #call, cudaGetErrorString(_e), cudaGetErrorName(_e)); \
            return ens_err(e, QGN_ERR_CUDA, _b);                                                    \
        }                                                                                           \
    } while (0)

bool fp32(const qgn_ens* e) { return e->precision == QGN_PREC_MIXED; }

int tv_of(const qgn_ens* e, int tp) {
    return fp32(e) ? ens_variant<float2>(tp, e->variant[tp]) : ens_variant<double2>(tp, e->variant[tp]);
}
int variant_count(const qgn_ens* e, int tp) {
    return fp32(e) ? ens_variant_count<float2>(tp) : ens_variant_count<double2>(tp);
}

int total_of(const qgn_ens* e, int pass) { return e->h_start[(size_t)pass * (e->mem.size() + 1) + e->mem.size()]; }

TileTab tab_of(const qgn_ens* e, int pass) {
    return TileTab{e->d_start + (size_t)pass * (e->mem.size() + 1), e->d_map + e->map_at[pass], total_of(e, pass)};
}

int grid_for(const qgn_ens* e, int pass, int tp) {
    const int total = total_of(e, pass);
    if (tp < 0 || e->grid_mode[tp] == 0) return std::max(1, total);
    return std::max(1, std::min(total, e->sms * e->grid_mode[tp]));
}

void build_tables(qgn_ens* e) {
    const size_t nm = e->mem.size();
    e->h_start.assign((size_t)EP_COUNT * (nm + 1), 0);
    e->h_map.clear();
    e->tables_new = true;
    for (int pass = 0; pass < EP_COUNT; ++pass) {
        if (pass == EP_XPASS) continue;
        int tv = 0;
        if (pass == EP_YINV) tv = tv_of(e, TP_YINV);
        if (pass == EP_YFWD) tv = tv_of(e, TP_YFWD);
        int* st = &e->h_start[(size_t)pass * (nm + 1)];
        e->map_at[pass] = (int)e->h_map.size();
        for (size_t m = 0; m < nm; ++m) {
            st[m + 1] = st[m] + member_tiles(e->mem[m]->g, pass, tv);
            e->h_map.resize(e->map_at[pass] + st[m + 1], (int)m);
        }
    }
    const int xtv = tv_of(e, TP_XPASS);
    e->h_xgroups.clear();
    for (qgn_ens::XGroup& x : e->xgroups) {
        x.table = (int)e->h_xgroups.size();
        e->h_xgroups.insert(e->h_xgroups.end(), x.members.begin(), x.members.end());
        x.map_at = (int)e->h_map.size();
        int sum = 0;
        for (size_t i = 0; i < x.members.size(); ++i) {
            e->h_xgroups.push_back(sum);
            sum += member_tiles(e->mem[x.members[i]]->g, EP_XPASS, xtv);
            e->h_map.resize(x.map_at + sum, (int)i);
        }
        e->h_xgroups.push_back(sum);
        x.tiles = sum;
    }
}

// the grid sizes of the members, largest first (the tail of a large launch costs the most)
void group_members(qgn_ens* e) {
    for (size_t m = 0; m < e->mem.size(); ++m) {
        const Geom& g = e->mem[m]->g;
        auto it = std::find_if(e->xgroups.begin(), e->xgroups.end(),
                               [&](const qgn_ens::XGroup& x) { return x.nx == g.nx && x.ny == g.ny; });
        if (it == e->xgroups.end()) {
            qgn_ens::XGroup x;
            x.nx = g.nx;
            x.ny = g.ny;
            e->xgroups.push_back(x);
            it = e->xgroups.end() - 1;
        }
        it->members.push_back((int)m);
    }
    std::sort(e->xgroups.begin(), e->xgroups.end(), [](const qgn_ens::XGroup& a, const qgn_ens::XGroup& b) {
        return (long long)a.nx * a.ny * (1 << 12) + a.nx > (long long)b.nx * b.ny * (1 << 12) + b.nx;
    });
}

// the tables to the device, if they are not those of the last upload
int upload_tables(qgn_ens* e) {
    if (!e->tables_new) return QGN_OK;
    if (e->h_map.size() > e->map_cap) {   // (a captured graph holds the old address)
        if (e->gexec) {
            ECK(cudaStreamSynchronize(e->stream));
            cudaGraphExecDestroy(e->gexec);
            e->gexec = nullptr;
        }
        if (e->d_map) ECK(cudaFree(e->d_map));
        e->d_map = nullptr;
        e->map_cap = 0;
        ECK(cudaMalloc((void**)&e->d_map, sizeof(int) * e->h_map.size()));
        e->map_cap = e->h_map.size();
    }
    ECK(cudaMemcpyAsync(e->d_map, e->h_map.data(), sizeof(int) * e->h_map.size(), cudaMemcpyHostToDevice, e->stream));
    ECK(cudaMemcpyAsync(e->d_start, e->h_start.data(), sizeof(int) * e->h_start.size(), cudaMemcpyHostToDevice,
                        e->stream));
    ECK(cudaMemcpyAsync(e->d_xgroups, e->h_xgroups.data(), sizeof(int) * e->h_xgroups.size(), cudaMemcpyHostToDevice,
                        e->stream));
    e->tables_new = false;
    ++e->uploads;
    return QGN_OK;
}

// member table from the contexts' current buffers
void fill_members(qgn_ens* e) {
    const bool f = fp32(e);
    for (size_t m = 0; m < e->mem.size(); ++m) {
        qgn_ctx* c = e->mem[m];
        Buffers& b = c->b;
        EnsMember& M = e->h_mem[m];
        std::memset(&M, 0, sizeof(M));
        M.g = c->g;
        M.q = b.q;
        M.qc = b.qnew;
        M.err = b.err;
        for (int j = 0; j < 4; ++j) M.N[j] = b.N[j];
        M.Qs = b.Qs[1];
        M.psi = b.psi;
        M.hq = b.hq;
        M.hp = b.hp;
        M.hu = b.hu;
        M.hpp = b.hpp;
        M.hpd = b.hpd;
        M.twx = f ? (const void*)b.twx32 : (const void*)b.twx;
        M.twy = f ? (const void*)b.twy32 : (const void*)b.twy;
        M.twx64 = b.twx;
        M.twy64 = b.twy;
        M.lc = b.lc;
        M.mc = b.mc;
        M.sc = b.sc;
        M.TOL = c->p.TOL;
        M.dt_max = c->p.dt_max;
        M.max_rejects = c->p.max_rejects > 0 ? c->p.max_rejects : 64;
        M.need_fsal = (e->seen_version[m] != c->state_version) ? 1 : 0;
    }
}

// ---- launches -------------------------------------------------------------------------------------
template <class CT>
int launch_stage(qgn_ens* e, int s) {
    double bytes = 0.0;
    for (qgn_ctx* c : e->mem) bytes += (double)c->g.csize() * (16.0 + 2.0 * sizeof(CT) + (s == 3 ? 3 : (s ? 1 : 0)) * sizeof(CT));
    bool nz16 = false;
    for (qgn_ctx* c : e->mem) nz16 = nz16 || c->g.nz == 16;
    QGN_LAUNCH(KID_STAGE, bytes, e->stream,
               ::qgn::launch(nz16 ? k_ens_stage<CT, true> : k_ens_stage<CT, false>, grid_for(e, EP_POINT, -1), kPointTile, 0,
                             e->stream, e->d_mem, tab_of(e, EP_POINT), s));
    ECK(cudaGetLastError());
    return QGN_OK;
}

template <class CT, int TV>
int launch_yinv_tv(qgn_ens* e, int s, int grid) {
    constexpr int SM = yinv_smem<CT, TV>();
    ECK(smem_attr(k_ens_yinv<CT, TV>, SM));
    double bytes = 0.0;
    for (qgn_ctx* c : e->mem) bytes += sizeof(CT) * (2.0 * c->g.csize() + 3.0 * c->g.nz * c->g.ny * c->g.nkx);
    QGN_LAUNCH(KID_YINV, bytes, e->stream,
               ::qgn::launch(k_ens_yinv<CT, TV>, grid, tv_width(TV), SM, e->stream, e->d_mem, tab_of(e, EP_YINV), s));
    ECK(cudaGetLastError());
    return QGN_OK;
}

// dynamic shared memory that keeps at most k CTAs of `need` bytes each on an SM: the least size of which
// k + 1, with what the system reserves per CTA, do not fit (a CTA cannot have more than smem_cta, which
// leaves room for no second one)
int limited_smem(const qgn_ens* e, int need, int k) {
    constexpr int kUnit = 128;   // allocation granularity
    const int s = (e->smem_sm / (k + 1) - e->smem_reserved) / kUnit * kUnit + kUnit;
    return std::max(need, std::min(s, e->smem_cta));
}

// occupancy: the resident CTAs per SM instead of a launch
template <int N, class CT, int TV>
int launch_xgroup(qgn_ens* e, const qgn_ens::XGroup& x, int s, int* occupancy) {
    // one CTA per tile; k > 0 CTAs per SM are a limit on the resident ones, by their shared memory
    const int gm = e->grid_mode[TP_XPASS], ng = (int)x.members.size();
    const int SM = gm == 0 ? XCfg<N, false, CT, TV>::SMEM : limited_smem(e, XCfg<N, false, CT, TV>::SMEM, gm);
    ECK(smem_attr(k_ens_xpass<N, CT, TV>, SM));
    if (occupancy) {
        int n = 0;
        ECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ens_xpass<N, CT, TV>, 3 * tv_width(TV), SM));
        *occupancy = std::max(*occupancy, n);
        return QGN_OK;
    }
    double bytes = 0.0;
    for (int m : x.members) {
        const Geom& g = e->mem[m]->g;
        bytes += 5.0 * sizeof(CT) * g.nz * g.ny * g.nkx;
    }
    const int grid = std::max(1, x.tiles);
    const int* idx = e->d_xgroups + x.table;
    QGN_LAUNCH(KID_XPASS, bytes, e->stream,
               ::qgn::launch(k_ens_xpass<N, CT, TV>, grid, 3 * tv_width(TV), SM, e->stream, e->mem[x.members[0]]->g, e->d_mem,
                             idx, TileTab{idx + ng, e->d_map + x.map_at, x.tiles}, s));
    ECK(cudaGetLastError());
    return QGN_OK;
}

template <class CT, int TV>
int launch_xpass_tv(qgn_ens* e, int s, int* occupancy) {
    for (const qgn_ens::XGroup& x : e->xgroups) {
        int r = QGN_ERR_CONFIG;
        switch (x.nx) {
            case 128: r = launch_xgroup<128, CT, TV>(e, x, s, occupancy); break;
            case 256: r = launch_xgroup<256, CT, TV>(e, x, s, occupancy); break;
            case 512: r = launch_xgroup<512, CT, TV>(e, x, s, occupancy); break;
            default: break;
        }
        if (r != QGN_OK) return r;
    }
    return QGN_OK;
}

template <class CT, int TV>
int launch_yfwd_tv(qgn_ens* e, int s, int grid) {
    constexpr int SM = yfwd_smem<CT, TV>();
    ECK(smem_attr(k_ens_yfwd<CT, TV>, SM));
    double bytes = 0.0;
    for (qgn_ctx* c : e->mem) bytes += sizeof(CT) * c->g.nz * c->g.nkx * (2.0 * c->g.ny + 3.0 * c->g.nky);
    QGN_LAUNCH(KID_YFWD, bytes, e->stream,
               ::qgn::launch(k_ens_yfwd<CT, TV>, grid, tv_width(TV), SM, e->stream, e->d_mem, tab_of(e, EP_YFWD), s));
    ECK(cudaGetLastError());
    return QGN_OK;
}

// variant v of a pass: the I-th instantiation of the pass's list for I == v
template <class CT, size_t... I>
int launch_yinv_v(qgn_ens* e, int v, int s, std::index_sequence<I...>) {
    int r = QGN_ERR_CONFIG;
    const int grid = grid_for(e, EP_YINV, TP_YINV);
    (void)((v == (int)I ? (r = launch_yinv_tv<CT, ens_variant<CT>(TP_YINV, (int)I)>(e, s, grid), true) : false) || ...);
    return r;
}
template <class CT, size_t... I>
int launch_xpass_v(qgn_ens* e, int v, int s, std::index_sequence<I...>, int* occupancy = nullptr) {
    int r = QGN_ERR_CONFIG;
    (void)((v == (int)I ? (r = launch_xpass_tv<CT, ens_variant<CT>(TP_XPASS, (int)I)>(e, s, occupancy), true) : false) ||
           ...);
    return r;
}
template <class CT, size_t... I>
int launch_yfwd_v(qgn_ens* e, int v, int s, std::index_sequence<I...>) {
    int r = QGN_ERR_CONFIG;
    const int grid = grid_for(e, EP_YFWD, TP_YFWD);
    (void)((v == (int)I ? (r = launch_yfwd_tv<CT, ens_variant<CT>(TP_YFWD, (int)I)>(e, s, grid), true) : false) || ...);
    return r;
}

template <class CT>
int launch_pass(qgn_ens* e, int tp, int s) {
    const int v = e->variant[tp];
    if (tp == TP_YINV) return launch_yinv_v<CT>(e, v, s, std::make_index_sequence<ens_variant_count<CT>(TP_YINV)>{});
    if (tp == TP_XPASS) return launch_xpass_v<CT>(e, v, s, std::make_index_sequence<ens_variant_count<CT>(TP_XPASS)>{});
    return launch_yfwd_v<CT>(e, v, s, std::make_index_sequence<ens_variant_count<CT>(TP_YFWD)>{});
}

// CTAs of the x pass resident on an SM as it is launched now (the most of its launches)
template <class CT>
int xpass_occupancy(qgn_ens* e, int* occupancy) {
    *occupancy = 0;
    return launch_xpass_v<CT>(e, e->variant[TP_XPASS], 0, std::make_index_sequence<ens_variant_count<CT>(TP_XPASS)>{},
                              occupancy);
}

template <class CT>
int launch_rhs_all(qgn_ens* e, int s) {
    for (int tp = 0; tp < TP_COUNT; ++tp) {
        int r = launch_pass<CT>(e, tp, s);
        if (r != QGN_OK) return r;
    }
    return QGN_OK;
}

template <class CT>
int launch_fsal(qgn_ens* e) {
    int r = launch_stage<CT>(e, 0);
    if (r == QGN_OK) r = launch_rhs_all<CT>(e, 0);
    if (r != QGN_OK) return r;
    QGN_LAUNCH(KID_SCALAR, 0.0, e->stream, ::qgn::launch(k_ens_fsal_done, 1, 256, 0, e->stream, e->d_mem, (int)e->mem.size()));
    ECK(cudaGetLastError());
    return QGN_OK;
}

template <class CT>
int launch_attempt(qgn_ens* e, const cudaGraphConditionalHandle* loop) {
    for (int s = 1; s <= 3; ++s) {
        int r = launch_stage<CT>(e, s);
        if (r == QGN_OK) r = launch_rhs_all<CT>(e, s);
        if (r != QGN_OK) return r;
    }
    double eb = 0.0, yb = 0.0, xb = 0.0;
    for (qgn_ctx* c : e->mem) {
        eb += (double)c->g.csize() * (4.0 * sizeof(CT) + 16.0);
        yb += 16.0 * ((double)c->g.csize() + (double)c->g.nz * c->g.ny * c->g.nkx);
        xb += 16.0 * (double)c->g.nz * c->g.ny * c->g.nkx;
    }
    const int nm = (int)e->mem.size();
    QGN_LAUNCH(KID_LINCOMB, eb, e->stream,
               ::qgn::launch(k_ens_err<CT>, grid_for(e, EP_ELEM, -1), kPointTile, 0, e->stream, e->d_mem, tab_of(e, EP_ELEM)));
    ECK(cudaGetLastError());
    ECK(smem_attr(k_ens_yinv1, yinv1_smem()));
    QGN_LAUNCH(KID_YINV, yb, e->stream,
               ::qgn::launch(k_ens_yinv1, grid_for(e, EP_YINV1, -1), 128, yinv1_smem(), e->stream, e->d_mem, tab_of(e, EP_YINV1)));
    ECK(cudaGetLastError());
    ECK(smem_attr(k_ens_xinv1, xinv1_smem()));
    QGN_LAUNCH(KID_XINV1, xb, e->stream,
               ::qgn::launch(k_ens_xinv1, grid_for(e, EP_XINV1, -1), 128, xinv1_smem(), e->stream, e->d_mem, tab_of(e, EP_XINV1)));
    ECK(cudaGetLastError());
    QGN_LAUNCH(KID_SCALAR, 0.0, e->stream,
               ::qgn::launch(k_ens_ctrl, 1, 256, 0, e->stream, e->d_mem, nm, loop ? *loop : 0, loop ? 1 : 0, e->d_any));
    ECK(cudaGetLastError());
    return QGN_OK;
}

int attempt(qgn_ens* e, const cudaGraphConditionalHandle* loop) {
    QGN_NVTX("ensemble attempt");
    return fp32(e) ? launch_attempt<float2>(e, loop) : launch_attempt<double2>(e, loop);
}
int fsal(qgn_ens* e) { return fp32(e) ? launch_fsal<float2>(e) : launch_fsal<double2>(e); }

// ---- autotuner: per right-hand-side pass, the tile-width variant and grid size with the
// shortest event-timed launch on this ensemble (outputs are scratch: stage 1's RHS1 and
// half-transformed fields, which the first attempt overwrites) ------------------------------
int autotune(qgn_ens* e) {
    cudaEvent_t a, b;
    ECK(cudaEventCreate(&a));
    ECK(cudaEventCreate(&b));
    const bool timing = e->prof.timing;
    e->prof.timing = false;
    long long launches0[KID_COUNT];
    for (int k = 0; k < KID_COUNT; ++k) launches0[k] = e->prof.launches[k];
    int rc = QGN_OK;
    const int grid_modes[4] = {0, 2, 4, 8};
    for (int tp = 0; tp < TP_COUNT && rc == QGN_OK; ++tp) {
        if (e->pinned[tp]) continue;
        float best = 1e30f;
        int bv = kDefaultVariant, bg = 0;
        for (int v = 0; v < variant_count(e, tp) && rc == QGN_OK; ++v) {
            e->variant[tp] = v;
            build_tables(e);
            rc = upload_tables(e);
            for (int gm = 0; gm < 4 && rc == QGN_OK; ++gm) {
                e->grid_mode[tp] = grid_modes[gm];
                const int reps = 5;
                rc = fp32(e) ? launch_pass<float2>(e, tp, 1) : launch_pass<double2>(e, tp, 1);   // warm-up
                if (rc != QGN_OK) break;
                if (cudaEventRecord(a, e->stream) != cudaSuccess) { rc = QGN_ERR_CUDA; break; }
                for (int r = 0; r < reps && rc == QGN_OK; ++r)
                    rc = fp32(e) ? launch_pass<float2>(e, tp, 1) : launch_pass<double2>(e, tp, 1);
                if (rc != QGN_OK) break;
                if (cudaEventRecord(b, e->stream) != cudaSuccess || cudaEventSynchronize(b) != cudaSuccess) {
                    rc = QGN_ERR_CUDA;
                    break;
                }
                float ms = 0.f;
                cudaEventElapsedTime(&ms, a, b);
                ms /= reps;
                if (ms < best) {
                    best = ms;
                    bv = v;
                    bg = grid_modes[gm];
                }
            }
        }
        e->variant[tp] = bv;
        e->grid_mode[tp] = bg;
        e->tuned_ms[tp] = best;
    }
    e->prof.timing = timing;
    for (int k = 0; k < KID_COUNT; ++k) e->prof.launches[k] = launches0[k];
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (rc != QGN_OK) return rc == QGN_ERR_CUDA && e->last_error.empty() ? ens_err(e, rc, "autotune failed") : rc;
    build_tables(e);
    return upload_tables(e);
}

int add_while(qgn_ens* e, cudaGraphConditionalHandle h, cudaGraph_t* body) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    ECK(cudaStreamGetCaptureInfo(e->stream, &cs, nullptr, &graph, &deps, &nd));
    cudaGraphNodeParams np = {cudaGraphNodeTypeConditional};
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    ECK(cudaGraphAddNode(&node, graph, deps, nd, &np));
    ECK(cudaStreamUpdateCaptureDependencies(e->stream, &node, 1, cudaStreamSetCaptureDependencies));
    *body = np.conditional.phGraph_out[0];
    return QGN_OK;
}

// root: FSAL pass (members that need RHS0) -> WHILE(any active) { attempt }
int capture(qgn_ens* e) {
    cudaGraph_t root = nullptr;
    long long c0[KID_COUNT], c1[KID_COUNT], c2[KID_COUNT];
    const bool timing = e->prof.timing;
    e->prof.timing = false;
    auto run = [&]() -> int {
        ECK(cudaGraphCreate(&root, 0));
        cudaGraphConditionalHandle hloop;
        ECK(cudaGraphConditionalHandleCreate(&hloop, root, 1u, cudaGraphCondAssignDefault));
        for (int k = 0; k < KID_COUNT; ++k) c0[k] = e->prof.launches[k];
        ECK(cudaStreamBeginCaptureToGraph(e->stream, root, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        int r = fsal(e);
        cudaGraph_t wbody = nullptr;
        if (r == QGN_OK) r = add_while(e, hloop, &wbody);
        cudaGraph_t tmp = nullptr;
        ECK(cudaStreamEndCapture(e->stream, &tmp));
        if (r != QGN_OK) return r;
        for (int k = 0; k < KID_COUNT; ++k) c1[k] = e->prof.launches[k];
        ECK(cudaStreamBeginCaptureToGraph(e->stream, wbody, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
        r = attempt(e, &hloop);
        ECK(cudaStreamEndCapture(e->stream, &tmp));
        if (r != QGN_OK) return r;
        for (int k = 0; k < KID_COUNT; ++k) c2[k] = e->prof.launches[k];
        ECK(cudaGraphInstantiate(&e->gexec, root, 0));
        return QGN_OK;
    };
    const int rc = run();
    e->prof.timing = timing;
    if (root) cudaGraphDestroy(root);
    for (int k = 0; k < KID_COUNT; ++k) {
        e->g_root[k] = c1[k] - c0[k];
        e->g_body[k] = c2[k] - c1[k];
        e->prof.launches[k] = c0[k];
    }
    return rc;
}

int read_member_scalars(qgn_ens* e, std::vector<DevScalars>& out) {
    out.resize(e->mem.size());
    for (size_t m = 0; m < e->mem.size(); ++m)
        ECK(cudaMemcpyAsync(&out[m], e->mem[m]->b.sc, sizeof(DevScalars), cudaMemcpyDeviceToHost, e->stream));
    ECK(cudaStreamSynchronize(e->stream));
    return QGN_OK;
}

}  // namespace

extern "C" {

int qgn_ens_create(qgn_ctx* const* members, int nmembers, int precision, qgn_ens** out) {
    if (!out) return QGN_ERR_ARG;
    *out = nullptr;
    if (!members || nmembers < 1 || nmembers > 4096) return QGN_ERR_ARG;
    if (precision != QGN_PREC_FP64 && precision != QGN_PREC_MIXED) return QGN_ERR_CONFIG;
    for (int m = 0; m < nmembers; ++m) {
        const qgn_ctx* c = members[m];
        if (!c) return QGN_ERR_ARG;
        if (c->scheme != QGN_SCHEME_BSRK3 || c->precision != QGN_PREC_FP64) return QGN_ERR_CONFIG;
        const int nx = c->g.nx, ny = c->g.ny;
        auto ok = [](int n) { return n == 128 || n == 256 || n == 512; };
        if (!ok(nx) || !ok(ny) || c->p.C_d != 0.0) return QGN_ERR_CONFIG;
        if (!(c->g.nz >= 2 && c->g.nz <= 8) && c->g.nz != 16) return QGN_ERR_CONFIG;
        if (c->device != members[0]->device) return QGN_ERR_CONFIG;
        for (int k = 0; k < m; ++k)
            if (members[k] == c) return QGN_ERR_ARG;
    }
    qgn_ens* e = new (std::nothrow) qgn_ens();
    if (!e) return QGN_ERR_CUDA;
    e->mem.assign(members, members + nmembers);
    e->seen_version.assign(nmembers, -1);
    e->precision = precision;
    e->device = members[0]->device;
    e->h_mem.resize(nmembers);
    e->graphs_off = std::getenv("QGN_NO_GRAPHS") != nullptr;
    auto fail = [&](int code) {
        qgn_ens_destroy(e);
        return code;
    };
    if (cudaSetDevice(e->device) != cudaSuccess) return fail(QGN_ERR_CUDA);
    const std::pair<int*, cudaDeviceAttr> attrs[] = {{&e->sms, cudaDevAttrMultiProcessorCount},
                                                     {&e->smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor},
                                                     {&e->smem_cta, cudaDevAttrMaxSharedMemoryPerBlockOptin},
                                                     {&e->smem_reserved, cudaDevAttrReservedSharedMemoryPerBlock}};
    for (const auto& a : attrs)
        if (cudaDeviceGetAttribute(a.first, a.second, e->device) != cudaSuccess) return fail(QGN_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(QGN_ERR_CUDA);
    if (cudaMalloc((void**)&e->d_mem, sizeof(EnsMember) * nmembers) != cudaSuccess) return fail(QGN_ERR_CUDA);
    if (cudaMalloc((void**)&e->d_start, sizeof(int) * (size_t)EP_COUNT * (nmembers + 1)) != cudaSuccess)
        return fail(QGN_ERR_CUDA);
    group_members(e);
    // a group of n members has 2 n + 1 entries
    if (cudaMalloc((void**)&e->d_xgroups, sizeof(int) * (2 * (size_t)nmembers + e->xgroups.size())) != cudaSuccess)
        return fail(QGN_ERR_CUDA);
    if (cudaMalloc((void**)&e->d_any, sizeof(int)) != cudaSuccess) return fail(QGN_ERR_CUDA);
    if (cudaMallocHost((void**)&e->h_any, sizeof(int)) != cudaSuccess) return fail(QGN_ERR_CUDA);
    build_tables(e);
    *out = e;
    return QGN_OK;
}

int qgn_ens_advance(qgn_ens* e, int nsteps) {
    QGN_NVTX("qgn_ens_advance");
    if (!e) return QGN_ERR_ARG;
    if (nsteps < 0) return ens_err(e, QGN_ERR_ARG, "nsteps < 0");
    EnsProfScope ps_(e);
    ECK(cudaSetDevice(e->device));
    const int nm = (int)e->mem.size();
    // members' own work (state uploads) precedes the ensemble's
    for (qgn_ctx* c : e->mem) ECK(cudaStreamSynchronize(c->stream));
    fill_members(e);
    ECK(cudaMemcpyAsync(e->d_mem, e->h_mem.data(), sizeof(EnsMember) * nm, cudaMemcpyHostToDevice, e->stream));
    int rc = upload_tables(e);
    if (rc != QGN_OK) return rc;
    QGN_LAUNCH(KID_SCALAR, 0.0, e->stream, ::qgn::launch(k_ens_arm, (nm + 255) / 256, 256, 0, e->stream, e->d_mem, nm, nsteps));
    ECK(cudaGetLastError());
    std::vector<DevScalars> s0, s1;
    if (!e->tuned && nsteps > 0) {
        // RHS0 with the default tiles, then tune on real fields
        rc = fsal(e);
        if (rc != QGN_OK) return rc;
        if (!std::getenv("QGN_NO_AUTOTUNE")) {
            rc = autotune(e);
            if (rc != QGN_OK) return rc;
        }
        e->tuned = true;
    }
    const bool use_graph = !e->graphs_off && !e->prof.timing;
    if (use_graph && !e->gexec) {
        rc = capture(e);
        if (rc != QGN_OK) {
            if (e->gexec) {
                cudaGraphExecDestroy(e->gexec);
                e->gexec = nullptr;
            }
            cudaGetLastError();
            e->graphs_off = true;
        }
    }
    rc = read_member_scalars(e, s0);
    if (rc != QGN_OK) return rc;
    if (nsteps > 0) {
        if (use_graph && e->gexec) {
            ECK(cudaGraphLaunch(e->gexec, e->stream));
        } else {
            rc = fsal(e);
            if (rc != QGN_OK) return rc;
            // bounded: every member halts after max_rejects consecutive rejections
            long long guard = 0;
            long long limit = 0;
            for (const EnsMember& M : e->h_mem) limit += (long long)nsteps * (M.max_rejects + 1);
            for (;;) {
                rc = attempt(e, nullptr);
                if (rc != QGN_OK) return rc;
                ECK(cudaMemcpyAsync(e->h_any, e->d_any, sizeof(int), cudaMemcpyDeviceToHost, e->stream));
                ECK(cudaStreamSynchronize(e->stream));
                e->prof.harvest();
                if (!*e->h_any || ++guard > limit) break;
            }
        }
    }
    rc = read_member_scalars(e, s1);
    if (rc != QGN_OK) return rc;
    if (use_graph && e->gexec && nsteps > 0) {
        // every attempt covers all members: the body ran as often as the busiest member attempted
        long long body_runs = 0;
        for (int m = 0; m < nm; ++m) body_runs = std::max(body_runs, s1[m].attempts - s0[m].attempts);
        for (int k = 0; k < KID_COUNT; ++k) e->prof.launches[k] += e->g_root[k] + body_runs * e->g_body[k];
    }
    // the device table holds the swapped state / RHS0 pointers: hand them back to the members
    ECK(cudaMemcpyAsync(e->h_mem.data(), e->d_mem, sizeof(EnsMember) * nm, cudaMemcpyDeviceToHost, e->stream));
    ECK(cudaStreamSynchronize(e->stream));
    e->prof.harvest();
    int first_bad = -1;
    for (int m = 0; m < nm; ++m) {
        qgn_ctx* c = e->mem[m];
        const EnsMember& M = e->h_mem[m];
        c->b.q = M.q;
        c->b.qnew = M.qc;
        c->b.N[0] = static_cast<double2*>(M.N[0]);
        c->b.N[3] = static_cast<double2*>(M.N[3]);
        c->b.Qs[0] = c->b.q;
        // an FP64 ensemble leaves a valid FP64 RHS0 for the member's own BSRK3 steps
        // (and none after a wait that ran out: RHS0 may be what lost it)
        c->first_call = fp32(e) || M.need_fsal != 0 || (s1[m].halt && s1[m].status == QGN_ERR_CUDA);
        e->seen_version[m] = c->state_version;
        if (s1[m].halt) {
            c->halted = true;
            if (first_bad < 0) first_bad = m;
        }
    }
    if (first_bad >= 0) {
        char buf[160];
        std::snprintf(buf, sizeof(buf), "member %d halted: %s", first_bad,
                      s1[first_bad].status == QGN_ERR_NONFINITE ? "non-finite embedded error estimate"
                      : s1[first_bad].status == QGN_ERR_CUDA    ? "a bounded device wait ran out"
                                                                : "adaptive step rejected max_rejects times in a row");
        return ens_err(e, s1[first_bad].status ? s1[first_bad].status : QGN_ERR_CUDA, buf);
    }
    return QGN_OK;
}

int qgn_ens_tuning(qgn_ens* e, int pass, int* threads, int* ctas_per_sm, float* ms) {
    if (!e || pass < 0 || pass >= TP_COUNT) return QGN_ERR_ARG;
    const int w = tv_width(tv_of(e, pass));
    if (threads) *threads = pass == TP_XPASS ? 3 * w : w;
    if (ctas_per_sm) *ctas_per_sm = e->grid_mode[pass];
    if (ms) *ms = e->tuned_ms[pass];
    return QGN_OK;
}

int qgn_ens_fft_radix(qgn_ens* e, int pass, int* elements_per_thread) {
    if (!e || !elements_per_thread || pass < 0 || pass >= TP_COUNT) return QGN_ERR_ARG;
    const int r = tv_radix(tv_of(e, pass));
    *elements_per_thread = r ? r : 16;
    return QGN_OK;
}

int qgn_ens_set_tiles(qgn_ens* e, int pass, int threads, int elements_per_thread, int ctas_per_sm) {
    if (!e || pass < 0 || pass >= TP_COUNT || ctas_per_sm < 0 || ctas_per_sm > 64) return QGN_ERR_ARG;
    const int w = pass == TP_XPASS ? threads / 3 : threads;
    if (pass == TP_XPASS && threads % 3 != 0) return ens_err(e, QGN_ERR_CONFIG, "x-pass threads: three slot groups");
    for (int v = 0; v < variant_count(e, pass); ++v) {
        const int tv = fp32(e) ? ens_variant<float2>(pass, v) : ens_variant<double2>(pass, v);
        if (tv_width(tv) == w && (tv_radix(tv) ? tv_radix(tv) : 16) == elements_per_thread) {
            e->variant[pass] = v;
            e->grid_mode[pass] = ctas_per_sm;
            e->pinned[pass] = true;
            e->tuned_ms[pass] = 0.f;
            build_tables(e);
            if (e->gexec) {   // the captured graph holds the old launches
                ECK(cudaStreamSynchronize(e->stream));
                cudaGraphExecDestroy(e->gexec);
                e->gexec = nullptr;
            }
            return QGN_OK;
        }
    }
    return ens_err(e, QGN_ERR_CONFIG, "no tile variant with these threads and elements per thread");
}

int qgn_ens_debug_residency(qgn_ens* e, int* ctas_per_sm) {
    if (!e || !ctas_per_sm) return QGN_ERR_ARG;
    ECK(cudaSetDevice(e->device));
    return fp32(e) ? xpass_occupancy<float2>(e, ctas_per_sm) : xpass_occupancy<double2>(e, ctas_per_sm);
}

int qgn_ens_debug_uploads(qgn_ens* e, int* count) {
    if (!e || !count) return QGN_ERR_ARG;
    *count = e->uploads;
    return QGN_OK;
}

int qgn_ens_profile_enable(qgn_ens* e, int on) {
    if (!e) return QGN_ERR_ARG;
    e->prof.reset();
    e->prof.timing = on != 0;
    return QGN_OK;
}

int qgn_ens_profile_read(qgn_ens* e, int kernel, double* ms, double* bytes, long long* timed, long long* launches) {
    if (!e || kernel < 0 || kernel >= KID_COUNT) return QGN_ERR_ARG;
    e->prof.harvest();
    if (ms) *ms = e->prof.total_ms[kernel];
    if (bytes) *bytes = e->prof.bytes[kernel];
    if (timed) *timed = e->prof.timed[kernel];
    if (launches) *launches = e->prof.launches[kernel];
    return QGN_OK;
}

int qgn_ens_stream(qgn_ens* e, void** stream) {
    if (!e || !stream) return QGN_ERR_ARG;
    *stream = e->stream;
    return QGN_OK;
}

const char* qgn_ens_last_error(qgn_ens* e) { return e ? e->last_error.c_str() : "NULL ensemble"; }

int qgn_ens_destroy(qgn_ens* e) {
    if (!e) return QGN_OK;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (e->gexec) cudaGraphExecDestroy(e->gexec);
    e->prof.release();
    if (e->d_mem) cudaFree(e->d_mem);
    if (e->d_start) cudaFree(e->d_start);
    if (e->d_xgroups) cudaFree(e->d_xgroups);
    if (e->d_map) cudaFree(e->d_map);
    if (e->d_any) cudaFree(e->d_any);
    if (e->h_any) cudaFreeHost(e->h_any);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return QGN_OK;
}

}  // extern "C"
