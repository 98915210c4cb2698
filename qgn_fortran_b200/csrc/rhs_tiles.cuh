// rhs_tiles.cuh -- per-tile bodies of the spectral right-hand side passes (see rhs_kernels.cu).
//
// Each body transforms one tile (a group of kx columns or of row pairs of one layer) whose
// coordinates the caller passes, so the same code serves the single-field launches
// (tile = blockIdx) and the ensemble launches, where a table maps a CTA to a member and tile.
// Bodies synchronise the whole CTA: every thread of the CTA must call them with its thread index.
#pragma once
#include "qgn_internal.cuh"
#include "fft.cuh"

#include <cuda.h>        // CUtensorMap (type only)
#include <cuda_bf16.h>

namespace qgn {

// ------------------------------------------------------------------------------------
// Tile shapes
// ------------------------------------------------------------------------------------
__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int cmin(int a, int b) { return a < b ? a : b; }

// slot stride (in elements) of a padded transform such that slot*stride spreads the bank
// groups of one shared-memory wavefront: W = 128 bytes / element size elements per wavefront
// (8 for double2, 16 for float2); target is the stride's residue mod W.
__host__ __device__ constexpr int slot_stride(int N, int target, int elem_bytes = 16, int tp = 16) {
    return (N + N / tp) + ((target - ((N + N / tp) % (128 / elem_bytes))) + (128 / elem_bytes)) % (128 / elem_bytes);
}
// residue for `slots` lane-interleaved slots: consecutive threads hit different slots
__host__ __device__ constexpr int interleave_target(int slots, int elem_bytes) {
    return slots >= 128 / elem_bytes ? 1 : (128 / elem_bytes) / slots;
}

// minimum resident CTAs for __launch_bounds__ such that a thread keeps up to maxregs registers
__host__ __device__ constexpr int minb(int threads, int maxregs = 128) {
    return cmax(1, cmin(8, 65536 / (threads * maxregs)));
}
// register budget per thread: an FP32 transform holds half the register bytes of an FP64 one
template <class CT>
__host__ __device__ constexpr int regcap(int fp64 = 128, int fp32 = 64) { return sizeof(CT) == 16 ? fp64 : fp32; }

// y-pass tiles: TKX kx columns per CTA, lane-interleaved (slot = tid % TKX) so that one
// warp touches 8 consecutive y rows of TKX adjacent columns: 16*TKX-byte segments in the
// half-transformed row layout, 128-byte segments in the compact column layout.
// The last parameter of each config selects a tile-width variant: 0 is the tuned default of
// the single-field launches; a non-zero value is the CTA size in threads (per slot group for
// the x pass), the same for every transform length, which lets one launch cover fields of
// different sizes (ensembles).
// elements per thread of an x transform (fft.cuh): 32 for the 512-point and longer transforms of
// the single-field x pass (two radix passes instead of three, each transform of up to 1024 points in
// one warp: the FP32 x pass ran 9 % faster, the FP64 one cut the 1024^2 x 8 step by 2 % despite 168
// registers), 16 otherwise.  2048 points take two warps and a third, radix-2 pass, which is fused with
// the second by shuffles (fft_pass_tail2, interleave 1): the 2048^2 x 16 x pass took 1061 us in FP64 and 511 us in
// FP32 with 16 elements and block barriers between all passes, 839 and 470 us this way.  The y passes
// keep 16 in FP32: their CTAs interleave columns across warps, and at 32 elements they had half the
// threads per column and ran 1.3-1.7x slower on B200.
// A non-zero tile-variant code carries the CTA width in its low 16 bits and, above them, the
// elements per thread of its transforms (8, 16 or 32; 0 there means 16): the ensemble's
// autotuner searches both.
__host__ __device__ constexpr int tv_width(int tv) { return tv & 0xFFFF; }
__host__ __device__ constexpr int tv_radix(int tv) { return tv >> 16; }
__host__ __device__ constexpr int tv_make(int width, int radix) { return width | (radix << 16); }
template <class CT, int N, int TV>
__host__ __device__ constexpr int fft_tp() {
    return TV == 0 ? ((N >= 512) ? 32 : 16) : (tv_radix(TV) ? tv_radix(TV) : 16);
}
// elements per thread of a y transform: 8 for the FP64 512- and 1024-point columns of the
// single-field launches, 16 otherwise.  Half the registers per thread (64, two 512-thread CTAs
// per SM) doubles the resident warps of these latency-bound kernels at the price of a fourth
// radix pass at 1024 points: on B200 the 512^2 step ran 11 % and the 1024^2 step 1 % faster.
// Columns per CTA (TKX) in FP64: at 2048 points a tile of the usual width is a 1024-thread CTA, alone on
// its SM; two columns of 16 elements per thread (y-inverse) and one (y-forward, whose rows come by
// tensor-map copies, so narrow pieces cost no L1 wavefronts) are 603 -> 477 us and 516 -> 411 us for
// 2048^2 x 16.  One column also suits the 1024-point y-forward (59.2 -> 55.5 us for 1024^2 x 8) but not
// the 512-point one (45.7 -> 48.8 us for 512^2 x 32); two in the y-inverse of 1024 points are slower
// (62.7 -> 68.4 us: its row stores fall to 32-byte pieces), as in the FP32 one of 2048 (274 -> 319 us).
// QGN_Y_TP64 (build-time tuning knob, default 8) overrides the FP64 value.
#ifndef QGN_Y_TP64
#define QGN_Y_TP64 8
#endif
template <class CT, int N, int TV>
__host__ __device__ constexpr int fft_tp_y() {
    return TV == 0 ? ((sizeof(CT) == 16 && N >= 512 && N < 2048) ? QGN_Y_TP64 : 16) : (tv_radix(TV) ? tv_radix(TV) : 16);
}
// Row pairs per CTA of the single-field x pass with one warp per transform (a build-time tuning
// knob).  One row pair (three warps, 96 threads, four CTAs per SM at 168 registers) couples only
// the three warps of a pair at the barrier between the inverse and forward transforms: the
// FP64 1024^2 x 8 x pass ran 7 % faster on B200 than with two row pairs per CTA.
#ifndef QGN_X_ROWPAIRS
#define QGN_X_ROWPAIRS 1
#endif

template <int NY, class CT = double2, int TV = 0>
struct YInvCfg {
    static constexpr int TP = fft_tp_y<CT, NY, TV>();
    static constexpr int G = FFTShape<NY, TP>::G;
    static constexpr int TKX = TV == 0 ? (NY >= 2048 && sizeof(CT) == 16 ? 2 : cmin(cmax(4, 128 / G), 16)) : cmax(1, tv_width(TV) / G);
    static constexpr int THREADS = TKX * G;
    static constexpr int TS = slot_stride(NY, interleave_target(TKX, (int)sizeof(CT)), (int)sizeof(CT), TP);
    static constexpr int SMEM = TKX * TS * (int)sizeof(CT);
    // de-interleaved output rows (yinv_tile): odd rows start at HY.  A wavefront holds W
    // elements, LP = W/TKX consecutive rows of each slot; HY = NY/2 + LP/2 puts their even and
    // odd halves on distinct bank groups.
    static constexpr int LP = cmax(1, (128 / (int)sizeof(CT)) / TKX);
    static constexpr int HY = NY / 2 + LP / 2;
    static_assert(2 * HY <= TS, "de-interleaved rows fit the slot");
};

template <int NX, bool DRAG, class CT = double2, int TV = 0>
struct XCfg {
    static constexpr int TP = fft_tp<CT, NX, TV>();
    static constexpr int G = FFTShape<NX, TP>::G;
    static constexpr int RP = (TV == 0 && G == 32) ? QGN_X_ROWPAIRS : cmax(1, (TV == 0 ? 64 : tv_width(TV)) / G);   // row pairs per CTA
    static constexpr int SP = 3;                        // slots per row pair
    static constexpr int THREADS = SP * RP * G;
    static constexpr int TS = slot_stride(NX, 2, (int)sizeof(CT), TP);
    static constexpr int SMEM = SP * RP * TS * (int)sizeof(CT);
};

template <int NY, bool DRAG, class CT = double2, int TV = 0>
struct YFwdCfg {
    static constexpr int TP = fft_tp_y<CT, NY, TV>();
    static constexpr int G = FFTShape<NY, TP>::G;
    // tid ^ TKX stays in the warp
    static constexpr int TKX = TV == 0 ? (NY >= 1024 && sizeof(CT) == 16 ? 1 : cmin(cmax(2, 64 / G), 16)) : cmin(cmax(1, tv_width(TV) / (2 * G)), 16);
    static constexpr int SLOTS = 2 * TKX;
    static constexpr int THREADS = SLOTS * G;
    static constexpr int TS = slot_stride(NY, interleave_target(SLOTS, (int)sizeof(CT)), (int)sizeof(CT), TP);
    static constexpr int SMEM = SLOTS * TS * (int)sizeof(CT);
};

// ------------------------------------------------------------------------------------
// Modal inversion: GetPsi (QGN_Module.f90:315-341) at every kept mode, all layers per thread
// ------------------------------------------------------------------------------------
template <int NZ>
__device__ __forceinline__ void modal_invert(const double* __restrict__ proj, const double* __restrict__ back,
                                             const double* __restrict__ ev, double Htot, int nz, double k2,
                                             bool mean_mode, const double2* qv, double2* pv) {
    constexpr int NZC = NZ > 0 ? NZ : kMaxNZ;
    const int n = NZ > 0 ? NZ : nz;
    double2 pm[NZC];
#pragma unroll
    for (int k = 0; k < NZC; ++k) {
        if (k < n) {
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll
            for (int kk = 0; kk < NZC; ++kk) {
                if (kk < n) {
                    double c = proj[k * n + kk];
                    acc.x += c * qv[kk].x;
                    acc.y += c * qv[kk].y;
                }
            }
            const double rden = 1.0 / ((-k2 + ev[k]) * Htot);
            pm[k] = mean_mode ? make_double2(0.0, 0.0) : make_double2(acc.x * rden, acc.y * rden);
        }
    }
#pragma unroll
    for (int k = 0; k < NZC; ++k) {
        if (k < n) {
            double2 acc = make_double2(0.0, 0.0);
#pragma unroll
            for (int kk = 0; kk < NZC; ++kk) {
                if (kk < n) {
                    double c = back[k * n + kk];
                    acc.x += pm[kk].x * c;
                    acc.y += pm[kk].y * c;
                }
            }
            pv[k] = acc;
        }
    }
}

// ------------------------------------------------------------------------------------
// Packed row pairs.  The x pass transforms rows y1 = 2p and y2 = 2p+1 of one field as one
// complex signal f1 + i f2 whose Hermitian extension is
//     A[k]      = F1[k] + i F2[k]               (0 <= k < nkx; Re parts only at k = 0)
//     A[nx - k] = conj(F1[k]) + i conj(F2[k])   (1 <= k < nkx)
// The y passes store exactly these two arrays per row pair: [nz][ny/2][2][nkxp] with slot
// 0 = A[k] and slot 1 = A[nx-k] (same bytes as two plain rows).  The x pass reads one value
// per element, and its forward transform writes P[k] and P[nx-k] of every row the same
// way, which the forward y pass splits into (uq)^ = (P[k] + conj P[nx-k])/2 and
// (vq)^ = (P[k] - conj P[nx-k])/(2i).
// ------------------------------------------------------------------------------------
template <class CT>
__device__ __forceinline__ CT pack_lo(CT f1, CT f2, bool k0) {
    return k0 ? cmk<CT>(f1.x, f2.x) : cmk<CT>(f1.x - f2.y, f1.y + f2.x);
}
template <class CT>
__device__ __forceinline__ CT pack_hi(CT f1, CT f2) {
    return cmk<CT>(f1.x + f2.y, f2.x - f1.y);
}

// Layout of the forward x transforms P[k] (part 0) and P[nx-k] (part 1) of every row y: the x
// pass's output, the forward y pass's input: rows [nz][ny][2 parts][nkxp], 2 nz ny nkxp elements.
// PT (the column kernels of small grids): columns [nz][nkxp][2 parts][ny], so that the x pass's stores,
// which nothing waits for, are the scattered side and a column is one contiguous load.
template <bool PT = false>
__host__ __device__ __forceinline__ size_t p_index(const Geom& g, int l, int y, int part, int k) {
    if (PT) return (((size_t)l * g.nkxp + k) * 2 + part) * g.ny + y;
    return ((size_t)l * g.ny + y) * 2 * g.nkxp + (size_t)part * g.nkxp + k;
}

// ------------------------------------------------------------------------------------
// Bulk-copy staging (cp.async.bulk, the untiled TMA copy) of contiguous global spans into shared
// memory, completing on an mbarrier.  Source and destination are 16-byte aligned and the sizes
// multiples of 16 bytes; a CTA copies from this GPU's own memory only, with no multicast.
// QGN_Y_BULK (build-time knob, default 1): the FP64 y-inverse stages its compact columns this way.
// ------------------------------------------------------------------------------------
#ifndef QGN_Y_BULK
#define QGN_Y_BULK 1
#endif
constexpr long long kBulkWaitLimit = 1LL << 22;   // polls of the mbarrier before the wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(bar)) : "memory");
    // the initialised barrier becomes visible to the async (bulk-copy) proxy
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void bar_inval(uint64_t* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// n elements from `first` requested into L2, widened to 16-byte boundaries (the fields' buffers hold 16
// bytes per element in either precision)
template <class CT>
__device__ __forceinline__ void prefetch_l2(const CT* first, int n) {
    const unsigned long long a = reinterpret_cast<unsigned long long>(first);
    const unsigned long long lo = a & ~15ull, hi = (a + (unsigned long long)n * sizeof(CT) + 15ull) & ~15ull;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(lo), "r"((uint32_t)(hi - lo)) : "memory");
}

// one box of a tensor map, its corner at (x, 0, y, l)
__device__ __forceinline__ void tensor_g2s(void* dst, const CUtensorMap* map, int x, int y, int l, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(0), "r"(y), "r"(l), "r"(smem_u32(bar))
        : "memory");
}
// bounded wait for phase `parity` of the barrier; false when it ran out
__device__ __forceinline__ bool bar_wait_bounded(uint64_t* bar, uint32_t parity) {
    const uint32_t a = smem_u32(bar);
    for (long long i = 0; i < kBulkWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// ------------------------------------------------------------------------------------
// yinv: inverse y transforms of kept columns into packed row pairs.
// NF = 3: (q -> pq, -i ky psi -> pu, i kx psi -> pv);  NF = 2: (q -> pq, psi -> pu);  NF = 1: (f -> pq).
// The first radix pass reads the compact column (zeros in the dealiased band) straight from HBM,
// or, in FP64 with a wait-flag in the geometry (QGN_Y_BULK), from the column's own shared-memory
// slot, where one bulk copy per column has staged it; the transformed column stays in shared
// memory, where a packing loop pairs rows y and y+1 and writes the two packed arrays with
// TKX-wide coalesced stores.
// ------------------------------------------------------------------------------------
template <int NY, int NF, class CT, int TV = 0>
// f_begin/f_end: the fields this CTA transforms (all NF by default; one each when a launch
// spreads the fields over CTAs)
__device__ __forceinline__ void yinv_tile(const Geom g, int tid, int bx, int l, const CT* __restrict__ q,
                                          const CT* __restrict__ psi, CT* __restrict__ pq, CT* __restrict__ pv,
                                          CT* __restrict__ pu, const CT* __restrict__ twy, int f_begin = 0,
                                          int f_end = NF) {
    using C = YInvCfg<NY, CT, TV>;
    using RT = typename CTraits<CT>::R;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    CT* sm = reinterpret_cast<CT*>(sm_raw);
    const int kx0 = bx * C::TKX;
    const int slot = tid % C::TKX, lane = tid / C::TKX;
    const int kx = kx0 + slot;
    const bool colok = kx < g.nkx;
    const size_t colbase = ((size_t)l * g.nkx + kx) * g.nky;
    const RT kxv = (RT)(g.dkx * kx);
    CT* xs = sm + slot * C::TS;
    NoIOT<CT> none;
#pragma unroll
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        if (f < f_begin || f >= f_end) continue;
        const CT* src = (f == 0) ? q : psi;
        CT* dst = (f == 0) ? pq : (f == 1 ? pu : pv);
        // the spectral derivative of field f at ky index j (QGN_Module.f90:223-224)
        auto deriv = [&](CT v, int j) -> CT {
            if (f == 1 && NF == 3) {   // u_hat = -i ky psi_hat
                const RT kyv = (RT)g.kyval(j);
                return cmk<CT>(kyv * v.y, -kyv * v.x);
            } else if (f == 2) {   // v_hat = i kx psi_hat
                return cmk<CT>(-kxv * v.y, kxv * v.x);
            }
            return v;
        };
        // the last pass writes rows y de-interleaved: even y at y/2, odd y at HY + y/2, so the
        // packing loop below reads consecutive offsets (free of bank-group conflicts; HY
        // offsets the odd half so that the last pass's stores are conflict-free too)
        auto omap = [](int y) { return (y & 1) * C::HY + (y >> 1); };
        bool staged = false;
        if constexpr (QGN_Y_BULK && sizeof(CT) == 16) {
            const int ncol = cmin(C::TKX, g.nkx - kx0);   // kept columns of this tile (>= 1)
            const size_t last = ((size_t)l * g.nkx + kx0 + ncol - 1) * g.nky + g.nky - 1;
            if (g.wait_err && in_bounds(g, last, g.csize())) {
                // one bulk copy per kept column into its slot (nky <= TS elements), thread 0 issues
                __shared__ __align__(8) uint64_t ybar;
                // this thread's earlier accesses to the slots are ordered before the copies' writes
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                if (tid == 0) bar_init(&ybar);
                __syncthreads();   // the barrier is initialised before anyone waits on it
                if (tid == 0) {
                    bar_expect_tx(&ybar, (uint32_t)(ncol * g.nky * (int)sizeof(CT)));
                    for (int c = 0; c < ncol; ++c)
                        bulk_g2s(sm + c * C::TS, src + ((size_t)l * g.nkx + kx0 + c) * g.nky,
                                 (uint32_t)(g.nky * (int)sizeof(CT)), &ybar);
                }
                if (!bar_wait_bounded(&ybar, 0)) {
                    atomicExch(g.wait_err, 1);            // the controller halts the run on it
                    bar_wait_bounded(&ybar, 0);           // once more for the copies still in flight
                }
                const CT* stage = xs;
                auto lds = [&](int j) -> CT {
                    const bool kept = (j < g.kylo) || (j >= g.kylo + g.kyshift);
                    if (!colok || !kept) return cmk<CT>(0.0, 0.0);
                    return deriv(stage[j < g.kylo ? j : j - g.kyshift], j);
                };
                // SRC_FN_SMEM: every thread has read the staged column before the first pass
                // overwrites the slot (block-wide barrier inside the pass)
                fft_fused<NY, +1, SRC_FN_SMEM, DST_SMEM_MAP, C::TP, false, C::TKX>(xs, lane, true, twy, lds, omap);
                if (tid == 0) bar_inval(&ybar);           // every waiter has passed the barrier
                staged = true;
            }
        }
        if (!staged) {
            auto ld = [&](int j) -> CT {
                const bool kept = (j < g.kylo) || (j >= g.kylo + g.kyshift);
                if (!colok || !kept) return cmk<CT>(0.0, 0.0);
                const size_t ci = colbase + (j < g.kylo ? j : j - g.kyshift);
                if (!in_bounds(g, ci, g.csize())) return cmk<CT>(0.0, 0.0);
                return deriv(src[ci], j);
            };
            fft_fused<NY, +1, SRC_FN, DST_SMEM_MAP, C::TP, false, C::TKX>(xs, lane, true, twy, ld, omap);
        }
        // pack rows (2p, 2p+1): e -> (pair p, column c); both arrays of a pair row per thread
        CT* dl = dst + (size_t)l * (NY / 2) * 2 * g.nkxp;
        for (int e = tid; e < (NY / 2) * C::TKX; e += C::THREADS) {
            const int p = e / C::TKX, c = e % C::TKX;
            const int k = kx0 + c;
            if (k >= g.nkxp) continue;
            const CT f1 = sm[c * C::TS + p], f2 = sm[c * C::TS + C::HY + p];
            const bool ok = k < g.nkx;
            const size_t ro = ((size_t)l * (NY / 2) + p) * 2 * g.nkxp;   // row pair p of layer l
            if (!in_bounds(g, ro + g.nkxp + k, g.hsize())) continue;
            CT* row = dl + (size_t)p * 2 * g.nkxp;
            // Re parts at kx = 0 and at the kx Nyquist column (kept only in the full-spectrum geometry)
            row[k] = ok ? pack_lo(f1, f2, k == 0 || 2 * k == g.nx) : cmk<CT>(0.0, 0.0);
            row[g.nkxp + k] = (ok && k > 0) ? pack_hi(f1, f2) : cmk<CT>(0.0, 0.0);
        }
        if (f + 1 < f_end) __syncthreads();   // the next field's first pass reuses the slots
    }
}

// ------------------------------------------------------------------------------------
// xpass: x transforms of row pairs.  c2r of the packed q1 + i q2, u1 + i u2, v1 + i v2
// (pairing two rows of one field keeps roundoff relative to that field; q and u differ by
// ~1e4 in these units), physical products formed inside the first pass of the forward
// transforms, r2c of p = uq + i vq per row, whose last pass writes P[k] and P[nx-k] for the
// kept kx straight to HBM.
//
// Quadratic drag (DRAG) adds the transforms of |u|u + i |u|v of the bottom layer (QGN_Module.f90:
// 284-292).  They are tiles of a layer of their own, l = nz, in the same launch: such a tile
// transforms u and v of the bottom layer once more (its q slot idles), turns them in place into
// |u|u and |u|v and runs the same forward transforms.  A second launch for the bottom layer alone,
// which it replaces, was 15 us of latency per right-hand side (64 CTAs at 512^2).
// ------------------------------------------------------------------------------------
template <int NX, bool DRAG, class CT, int TV = 0, bool PT = false>
__device__ __forceinline__ void xpass_tile(const Geom g, int tid, int bx, int layer, const CT* __restrict__ pq,
                                           const CT* __restrict__ pv, const CT* __restrict__ pu,
                                           CT* __restrict__ pp, CT* __restrict__ pd, const CT* __restrict__ twx) {
    using C = XCfg<NX, DRAG, CT, TV>;
    using RT = typename CTraits<CT>::R;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    CT* sm = reinterpret_cast<CT*>(sm_raw);
    const int npairs = g.ny / 2;
    const int nkx = g.nkx;
    const int slot = tid / C::G, lane = tid % C::G;
    const int r_of = slot / C::SP, s_of = slot % C::SP;
    const int rp = bx * C::RP + r_of;
    const bool pair_ok = rp < npairs;
    const bool drag = DRAG && layer == g.nz;   // this tile makes the drag fields of the bottom layer
    const int l = drag ? g.nz - 1 : layer;
    CT* base = sm + (r_of * C::SP) * C::TS;
    CT* xs = sm + slot * C::TS;

    // ---- inverse: slot 0 = q1+iq2, 1 = u1+iu2, 2 = v1+iv2
    const size_t fo = ((size_t)l * npairs + rp) * 2 * g.nkxp;   // row pair rp of layer l
    const CT* F = (s_of == 0 ? pq : (s_of == 1 ? pu : pv)) + fo;
    auto ld_inv = [&](int k) -> CT {
        if (k < nkx) return in_bounds(g, fo + k, g.hsize()) ? F[k] : cmk<CT>(0.0, 0.0);
        if (k > NX - nkx) return in_bounds(g, fo + g.nkxp + (NX - k), g.hsize()) ? F[g.nkxp + (NX - k)] : cmk<CT>(0.0, 0.0);
        return cmk<CT>(0.0, 0.0);
    };
    // the last pass stores the two rows apart, as real planes: row 2p at RT offset 0 of the
    // slot, row 2p+1 at RT offset TS, so that each forward transform below reads only its
    // own row (half the bytes of reading the packed complex values)
    RT* plane = reinterpret_cast<RT*>(xs);
    auto st_inv = [&](int x, CT v) {
        plane[x] = v.x;
        plane[C::TS + x] = v.y;
    };
    fft_fused<NX, +1, SRC_FN, DST_SMEM_STORE, C::TP, (C::G <= 32), (C::G > 32 && TV == 0 ? 1 : 0)>(xs, lane, pair_ok && !(drag && s_of == 0), twx,
                                                                     ld_inv, st_inv);

    // ---- forward: slot 0 = u1 q1 + i v1 q1, 1 = u2 q2 + i v2 q2 (grid/(nx*ny) scaling as in
    //      QGN_Module.f90:229-235); a drag tile |u1|u1 + i|u1|v1 and |u2|u2 + i|u2|v2
    const RT sc = (RT)g.inv_nxny;
    const RT sc2 = sc * sc;   // nx, ny are powers of two: u (q sc^2) == (u sc)(q sc) exactly
    // this slot's row in the planes of the q, u, v slots (RT offsets 0, 2 TS, 4 TS)
    const RT* rows = reinterpret_cast<const RT*>(base) + ((s_of & 1) ? C::TS : 0);
    if (drag) {   // u, v -> |u|u, |u|v in place (URMS, QGN_Module.f90:285)
        for (int e = tid; e < C::RP * 2 * NX; e += C::THREADS) {
            RT* pl = reinterpret_cast<RT*>(sm + (e / (2 * NX)) * C::SP * C::TS) + ((e / NX) & 1) * C::TS + e % NX;
            const RT uv = pl[2 * C::TS] * sc, vv = pl[4 * C::TS] * sc;
            const RT m = sqrt(uv * uv + vv * vv);
            pl[2 * C::TS] = m * uv;
            pl[4 * C::TS] = m * vv;
        }
        __syncthreads();
    }
    auto ld_fwd = [&](int x) -> CT {
        const RT qs = drag ? (RT)1 : rows[x] * sc2;
        return cmk<CT>(rows[2 * C::TS + x] * qs, rows[4 * C::TS + x] * qs);
    };
    const int y = 2 * rp + (s_of & 1);
    const int ol = drag ? 0 : l;                                                 // pd holds one layer
    const size_t olen = drag ? (size_t)g.ny * 2 * g.nkxp : 2 * g.hsize();   // pd, or pp
    CT* out = drag ? pd : pp;
    auto st_fwd = [&](int k, CT v) {
        if (k < nkx) {
            const size_t i = p_index<PT>(g, ol, y, 0, k);
            if (in_bounds(g, i, olen)) out[i] = v;
        } else if (k > NX - nkx) {
            const size_t i = p_index<PT>(g, ol, y, 1, NX - k);
            if (in_bounds(g, i, olen)) out[i] = v;
        }
    };
    fft_fused<NX, -1, SRC_FN_SMEM, DST_FN, C::TP, (C::G <= 32), (C::G > 32 && TV == 0 ? 1 : 0)>(xs, lane, pair_ok && s_of < 2, twx, ld_fwd, st_fwd);
}

// ------------------------------------------------------------------------------------
// yfwd: forward y transforms of uq, vq columns and assembly of the right-hand side.
// Slots are lane-interleaved: slot = tid % (2 TKX), slot = field*TKX + column.
//
// With a tensor map of the half-transformed rows (MAP) the tile -- TKX columns of both parts of every
// row, 2 TKX values per row -- is first copied into the slots' shared memory as [row][part][column] by
// the copy engine, and the first radix pass reads it there.  Plain loads of the rows take 16 or 32 bytes
// from each of 16 lines per warp (two columns), so the pass was bound by the L1's line rate: 38 % of
// its L1 wavefronts were these loads.  The staged form needs a fourth of them, and reads both parts
// instead of exchanging them by shuffles.  When the copies have landed, the columns of q and psi that
// the assembly will read are requested into L2, behind the transforms.  1024^2 x 8 FP64 66.1 -> 62.8 us
// staged -> 58.9 us with the request (63.9 us when it goes out before the copies), FP32 43.5 -> 39.7 ->
// 36.6 us, 2048^2 x 16 FP32 281 -> 255 -> 225 us, 512^2 x 32 FP64 55.8 -> 49.8 -> 45.9 us (B200).
// Without one (ensembles, small tiles) the first radix pass reads the rows straight from HBM.
// ------------------------------------------------------------------------------------
struct YfwdMaps {       // of hpp and, with drag, of hpd; use = 0: none (plain staging loads)
    CUtensorMap p, d;
    int use;
};

template <class CT>
__device__ __forceinline__ CT split_p(CT X, CT P1, int kx, int fld) {
    using RT = typename CTraits<CT>::R;
    const CT Y = kx == 0 ? cconj(X) : cconj(P1);
    return fld == 0 ? cmk<CT>((RT)0.5 * (X.x + Y.x), (RT)0.5 * (X.y + Y.y))
                    : cmk<CT>((RT)0.5 * (X.y - Y.y), -(RT)0.5 * (X.x - Y.x));
}

// the tile's columns of every row of layer l into sm as [NY][2][TKX]; bar: a barrier past the slots,
// fresh for each call (initialised and invalidated here)
template <int NY, int TKX, class CT>
__device__ __forceinline__ void stage_rows(const Geom& g, int tid, int threads, int kx0, int l, const CUtensorMap* map,
                                           bool use, const CT* __restrict__ P, size_t len, CT* sm, uint64_t* bar) {
    if (use) {
        constexpr int ROWS = NY < 256 ? NY : 256;   // rows per box
        // the slots' earlier accesses are ordered before the copies' writes
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        if (tid == 0) bar_init(bar);
        __syncthreads();
        if (tid == 0) {
            bar_expect_tx(bar, (uint32_t)(NY * 2 * TKX * (int)sizeof(CT)));
            for (int y = 0; y < NY; y += ROWS) tensor_g2s(sm + (size_t)y * 2 * TKX, map, 2 * kx0, y, l, bar);
        }
        if (!bar_wait_bounded(bar, 0)) {
            atomicExch(g.wait_err, 1);            // the controller halts the run on it
            bar_wait_bounded(bar, 0);             // once more for the copies still in flight
        }
    } else {
        for (int e = tid; e < NY * 2 * TKX; e += threads) {
            const int c = e % TKX, part = (e / TKX) % 2, y = e / (2 * TKX);
            const size_t i = p_index(g, l, y, part, kx0 + c);
            const bool ok = kx0 + c < g.nkx && in_bounds(g, i, len);
            sm[e] = ok ? P[i] : cmk<CT>(0.0, 0.0);
        }
        __syncthreads();
    }
}

// the thread of field fld loads part fld (P[k] for fld 0, P[nx-k] for fld 1) at index i and
// swaps it with its partner's, so each value is read once
template <class CT>
__device__ __forceinline__ CT unpack_pair(const CT* __restrict__ P, size_t i, int kx, int fld, bool ok, int partner) {
    CT mine = cmk<CT>(0.0, 0.0);
    if (ok && (fld == 0 || kx > 0)) mine = P[i];
    CT other;
    other.x = __shfl_xor_sync(0xffffffffu, mine.x, partner);
    other.y = __shfl_xor_sync(0xffffffffu, mine.y, partner);
    const CT X = fld == 0 ? mine : other;
    const CT Y = kx == 0 ? cconj(X) : cconj(fld == 0 ? other : mine);
    return fld == 0 ? cmk<CT>((typename CTraits<CT>::R)0.5 * (X.x + Y.x), (typename CTraits<CT>::R)0.5 * (X.y + Y.y))
                    : cmk<CT>((typename CTraits<CT>::R)0.5 * (X.y - Y.y), -(typename CTraits<CT>::R)0.5 * (X.x - Y.x));
}

template <int NY, bool DRAG, class CT, int TV = 0, bool MAP = false, bool PT = false>
__device__ __forceinline__ void yfwd_tile(const Geom g, int tid, int bx, int l, const LayerConst* __restrict__ lc,
                                          const CT* __restrict__ q, const CT* __restrict__ psi,
                                          const CT* __restrict__ pp, const CT* __restrict__ pd,
                                          CT* __restrict__ out, const CT* __restrict__ twy,
                                          const CT* __restrict__ extra = nullptr, const YfwdMaps* maps = nullptr) {
    static_assert(!(PT && (MAP || DRAG)), "columns come by plain loads, without drag");
    using C = YFwdCfg<NY, DRAG, CT, TV>;
    using RT = typename CTraits<CT>::R;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    CT* sm = reinterpret_cast<CT*>(sm_raw);
    const int kx0 = bx * C::TKX;
    const int slot = tid % C::SLOTS, lane = tid / C::SLOTS;
    const int fld = slot / C::TKX, c = slot % C::TKX;
    const bool colok = kx0 + c < g.nkx;
    const int nky = g.nky;
    const size_t colbase = (size_t)l * g.nkx;
    const bool bottom = (l == g.nz - 1);
    CT* xs = sm + slot * C::TS;
    // the last radix pass writes the transformed column unpadded (row y at y): the assembly
    // loops below read 8-16 consecutive rows per wavefront, which a pad element every TP rows
    // would split across one bank group twice
    auto omap = [](int y) { return y; };
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm_raw + C::SMEM);   // (MAP)
    auto ld_staged = [&](int y) -> CT {
        const CT X = sm[(2 * y) * C::TKX + c], P1 = sm[(2 * y + 1) * C::TKX + c];
        const CT v = split_p(X, P1, kx0 + c, fld);
        return colok ? v : cmk<CT>(0.0, 0.0);
    };

    if (DRAG && bottom) {
        // drag_hat = i ky (|u|u)^ - i kx (|u|v)^ on the bottom layer (QGN_Module.f90:284-292)
        auto ldd = [&](int y) -> CT {
            const size_t i = p_index(g, 0, y, fld, kx0 + c);
            const bool ok = colok && in_bounds(g, i, (size_t)g.ny * 2 * g.nkxp);
            return unpack_pair(pd, i, kx0 + c, fld, ok, C::TKX);
        };
        if constexpr (MAP) {
            stage_rows<NY, C::TKX>(g, tid, C::THREADS, kx0, 0, &maps->d, maps->use, pd, (size_t)g.ny * 2 * g.nkxp, sm, bar);
            fft_fused<NY, -1, SRC_FN_SMEM, DST_SMEM_MAP, C::TP, false, C::SLOTS>(xs, lane, true, twy, ld_staged, omap);
            if (maps->use && tid == 0) bar_inval(bar);   // every waiter has passed the barrier
        } else {
            fft_fused<NY, -1, SRC_FN, DST_SMEM_MAP, C::TP, false, C::SLOTS>(xs, lane, true, twy, ldd, omap);
        }
        const RT dc = (RT)lc->dragc;
        for (int e = tid; e < C::TKX * nky; e += C::THREADS) {
            const int cc = e / nky, m = e % nky;
            const int kx = kx0 + cc;
            if (kx >= g.nkx) continue;
            const int j = g.jfull(m);
            const RT kxv = (RT)(g.dkx * kx), kyv = (RT)g.kyval(j);
            const CT fu = sm[cc * C::TS + j], fv = sm[(C::TKX + cc) * C::TS + j];
            CT d = cmk<CT>(-kyv * fu.y, kyv * fu.x);        // i ky (|u|u)^
            d = cmk<CT>(d.x + kxv * fv.y, d.y - kxv * fv.x);      // - i kx (|u|v)^
            if (in_bounds(g, (colbase + kx) * nky + m, g.csize())) out[(colbase + kx) * nky + m] = cmk<CT>(dc * d.x, dc * d.y);
        }
        __syncthreads();
    }

    // the (uq)^ and (vq)^ slots of one column load P[k] and P[nx-k] respectively and swap
    // them with a shuffle (partner tid ^ TKX, same warp), so each value is read once
    auto ld = [&](int y) -> CT {
        const size_t i = p_index<PT>(g, l, y, fld, kx0 + c);
        const bool ok = colok && in_bounds(g, i, 2 * g.hsize());
        return unpack_pair(pp, i, kx0 + c, fld, ok, C::TKX);
    };
    if constexpr (MAP) {
        stage_rows<NY, C::TKX>(g, tid, C::THREADS, kx0, l, &maps->p, maps->use, pp, 2 * g.hsize(), sm, bar);
        const int ncol = cmin(C::TKX, g.nkx - kx0);
        if (tid >= 32 && tid < 34) prefetch_l2((tid == 32 ? q : psi) + (colbase + kx0) * nky, ncol * nky);
        fft_fused<NY, -1, SRC_FN_SMEM, DST_SMEM_MAP, C::TP, false, C::SLOTS>(xs, lane, true, twy, ld_staged, omap);
        if (maps->use && tid == 0) bar_inval(bar);
    } else {
        fft_fused<NY, -1, SRC_FN, DST_SMEM_MAP, C::TP, false, C::SLOTS>(xs, lane, true, twy, ld, omap);
    }

    const RT ub = (RT)lc->uBar[l], bq = (RT)lc->betaq[l];
    const RT ek = (RT)lc->ekman;
    const bool expl = lc->explicit_diss != 0;
    for (int e = tid; e < C::TKX * nky; e += C::THREADS) {
        const int cc = e / nky, m = e % nky;
        const int kx = kx0 + cc;
        if (kx >= g.nkx) continue;
        const int j = g.jfull(m);
        const RT kxv = (RT)(g.dkx * kx), kyv = (RT)g.kyval(j);
        const size_t idx = (colbase + kx) * nky + m;
        if (!in_bounds(g, idx, g.csize())) continue;
        const CT fuq = sm[cc * C::TS + j], fvq = sm[(C::TKX + cc) * C::TS + j];
        const CT qv = q[idx], pv = psi[idx];
        // jaco_hat = i kx uq_hat + i ky vq_hat  (QGN_Module.f90:244-247)
        const CT jac = cmk<CT>(-kxv * fuq.y - kyv * fvq.y, kxv * fuq.x + kyv * fvq.x);
        CT r = cmk<CT>(-jac.x, -jac.y);
        // - uBar i kx q_hat - (beta+qyBar) v_hat   (QGN_Module.f90:270-273)
        const RT uk = ub * kxv;
        const CT vh = cmk<CT>(-kxv * pv.y, kxv * pv.x);
        r = cmk<CT>(r.x + uk * qv.y, r.y - uk * qv.x);
        r = cmk<CT>(r.x - bq * vh.x, r.y - bq * vh.y);
        const RT k2 = kxv * kxv + kyv * kyv;
        if (expl) {   // QGN_Module.f90:275-280
            const RT k4 = k2 * k2, k8 = k4 * k4;
            const RT dcoef = (RT)lc->A2 * k2 + (RT)lc->A8 * k8;
            r = cmk<CT>(r.x - dcoef * qv.x, r.y - dcoef * qv.y);
        }
        if (bottom) {   // Ekman, QGN_Module.f90:282
            const RT ekk = ek * k2;
            r = cmk<CT>(r.x + ekk * pv.x, r.y + ekk * pv.y);
            if (DRAG) {
                const CT d = out[idx];
                r = cmk<CT>(r.x + d.x, r.y + d.y);
            }
        }
        if (extra) {   // an extra tendency on the kept modes (the learned closure's)
            const CT x = extra[idx];
            r = cmk<CT>(r.x + x.x, r.y + x.y);
        }
        if (kx == 0 && m == 0) r = cmk<CT>(0.0, 0.0);
        out[idx] = r;
    }
}

// ------------------------------------------------------------------------------------
// Single-field inverse 2-D transform: x c2r of row pairs with an epilogue
//   EPI 0: max |grid| (unnormalised) into sc->maxbits
//   EPI 1: physical field grid/(nx*ny) into out[nz][ny][nx]
// ------------------------------------------------------------------------------------
template <int NX, int TV = 0, class CT = double2>
struct X1Cfg {
    static constexpr int TP = 16;
    static constexpr int G = FFTShape<NX, TP>::G;
    static constexpr int RP = cmax(1, (TV == 0 ? 128 : TV) / G);
    static constexpr int THREADS = RP * G;
    static constexpr int TS = slot_stride(NX, 2, (int)sizeof(CT));
    static constexpr int SMEM = RP * TS * (int)sizeof(CT);
};

// CT = float2 (the mixed mode's error norm) supports EPI 0 only
template <int NX, int EPI, int TV = 0, class CT = double2>
// EPI 2 (the learned closure's input): channel chan of the NHWC BF16 tensor xout with
// cin_p channels per pixel, grid/(nx*ny) * scale[chan]
__device__ __forceinline__ void xinv1_tile(const Geom g, int bx, int l, const CT* __restrict__ hq,
                                           DevScalars* __restrict__ sc, double* __restrict__ outp,
                                           const CT* __restrict__ twx, const float* __restrict__ scale = nullptr,
                                           __nv_bfloat16* __restrict__ xout = nullptr, int cin_p = 0,
                                           int chan = 0) {
    static_assert(EPI == 0 || sizeof(CT) == 16, "FP32 rows: max only");
    using C = X1Cfg<NX, TV, CT>;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    CT* sm = reinterpret_cast<CT*>(sm_raw);
    __shared__ double smax[32];
    const int tid = threadIdx.x;
    const int npairs = g.ny / 2;
    const int nkx = g.nkx;
    const int slot = tid / C::G, lane = tid % C::G;
    const int rp = bx * C::RP + slot;
    const bool ok = rp < npairs;
    const CT* F = hq + ((size_t)l * npairs + rp) * 2 * g.nkxp;   // packed row pair
    auto ld = [&](int k) -> CT {
        if (k < nkx) return F[k];
        if (k > NX - nkx) return F[g.nkxp + (NX - k)];
        return cmk<CT>(0.0, 0.0);
    };
    double mx = 0.0;
    const size_t prow = ((size_t)l * g.ny + 2 * rp) * NX;
    auto st = [&](int x, CT a) {
        if constexpr (EPI == 0) {
            // NaN is kept as the largest value
            const double m1 = fabs((double)a.x), m2 = fabs((double)a.y);
            if (!(m1 == m1) || !(m2 == m2)) mx = __longlong_as_double(0x7ff8000000000000LL);
            else if (mx == mx) mx = fmax(mx, fmax(m1, m2));
        } else if constexpr (EPI == 1) {
            outp[prow + x] = a.x * g.inv_nxny;
            outp[prow + NX + x] = a.y * g.inv_nxny;
        } else {
            const size_t pix = (size_t)(2 * rp) * NX + x;
            const float sf = scale[chan];
            xout[pix * cin_p + chan] = __float2bfloat16_rn((float)(a.x * g.inv_nxny) * sf);
            xout[(pix + NX) * cin_p + chan] = __float2bfloat16_rn((float)(a.y * g.inv_nxny) * sf);
        }
    };
    fft_fused<NX, +1, SRC_FN, DST_FN, C::TP, (C::G <= 32)>(sm + slot * C::TS, lane, ok, twx, ld, st);
    if (EPI == 0) {
        // block max of non-negative doubles (NaN as the largest bit pattern)
        unsigned long long bits = (unsigned long long)__double_as_longlong(mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long ob = __shfl_xor_sync(0xffffffffu, bits, o);
            bits = ob > bits ? ob : bits;
        }
        if ((tid & 31) == 0) smax[tid >> 5] = __longlong_as_double((long long)bits);
        __syncthreads();
        if (tid < 32) {
            unsigned long long b2 = (tid < (C::THREADS + 31) / 32)
                                        ? (unsigned long long)__double_as_longlong(smax[tid]) : 0ULL;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                unsigned long long ob = __shfl_xor_sync(0xffffffffu, b2, o);
                b2 = ob > b2 ? ob : b2;
            }
            if (tid == 0) atomicMax(&sc->maxbits, b2);
        }
    }
}

}  // namespace qgn
