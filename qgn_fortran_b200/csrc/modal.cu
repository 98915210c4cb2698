// modal.cu -- GetPsi (QGN_Module.f90:315-341): psi = Modes diag(1/(-k^2 + EVals)) (H Modes)^T q / Htot
// at every kept mode, as two nz x nz contractions over the layers.
//
// Two forms, chosen by the layer count (launch_modal_any):
//   nz <= 8    k_modal<NZ>: one thread per mode holds the layers in registers and reads the
//              matrices from the constant bank; memory-bound (at nz = 8 on 1024^2, 59.5 MB in
//              14.4 us).
//   nz >= 9    k_modal_mma<NP>: the contractions on the FP64 matrix units (mma.m8n8k4.f64, the
//              widest FP64 form there is: tcgen05 has no FP64 kind), NP = nz rounded up to 8.
// One thread cannot hold more than 16 layers of q, the modal amplitudes and psi (3 nz complex
// doubles): the generic form kept them in local memory and took 117 us for 32 layers on 512^2,
// against 29.5 us here, and 42 us for 5 layers on 512 x 256 (in the explicit combinations),
// against 8.6 us.  At exactly 16 layers both fit, and it is the input that decides (2048^2, us):
// FP64 114.8 one-thread, 107.9 matrix units; FP32 110.0 one-thread, 115.1 matrix units, whose
// quarter-warps read 32-byte pieces of an FP32 field.  (On smaller grids the one-thread form's chain of
// products shows: FP32, 16 layers in it against 15 padded to 16 on the matrix units, events included, 64^2
// 11.5 / 8.6, 256^2 12.4 / 9.0, 512^2 15.0 / 14.5, 1024^2 34.6 / 33.4; the rule goes by the large grids.)
// 9 to 15 layers are padded to 16: FP32, in the generic form / here, 9 layers 64^2 30.5 / 8.7, 1024^2
// 140.9 / 31.7; 15 layers 39.1 / 8.6 and 212.4 / 33.4.
#include "qgn_internal.cuh"
#include "prof.cuh"
#include "rhs_tiles.cuh"

namespace qgn {

// stores of the two precisions
template <class T> struct ModalStore;
template <> struct ModalStore<double2> {
    __device__ static double2 put(double2 v) { return v; }
};
template <> struct ModalStore<float2> {
    __device__ static float2 put(double2 v) { return make_float2((float)v.x, (float)v.y); }
};

// TI: type of q; TO: type of psi.  COPY: q is also stored as TO into qcopy (the mixed mode's FP32
// copy of the state).
template <int NZ, class TI, class TO, bool COPY>
__global__ void __launch_bounds__(256, 2) k_modal(Geom g, const __grid_constant__ ModalParams<NZ> ma,
                                                  const TI* __restrict__ q, TO* __restrict__ psi,
                                                  TO* __restrict__ qcopy) {
    QGN_PDL_ENTRY();
    const size_t P = (size_t)g.nkx * g.nky;
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    const int kx = (int)((unsigned)p / (unsigned)g.nky), m = (int)((unsigned)p % (unsigned)g.nky);
    const double kxv = g.dkx * kx, kyv = g.kyval(g.jfull(m));
    const double k2 = kxv * kxv + kyv * kyv;
    double2 qv[NZ], pv[NZ];
#pragma unroll
    for (int k = 0; k < NZ; ++k) {
        const size_t i = (size_t)k * P + p;
        if (in_bounds(g, i, g.csize())) {
            const TI v = q[i];
            qv[k] = make_double2(v.x, v.y);
        } else {
            qv[k] = make_double2(0.0, 0.0);
        }
    }
    modal_invert<NZ>(ma.proj, ma.back, ma.ev, ma.Htot, NZ, k2, p == 0, qv, pv);
#pragma unroll
    for (int k = 0; k < NZ; ++k) {
        const size_t i = (size_t)k * P + p;
        if (!in_bounds(g, i, g.csize())) continue;
        psi[i] = ModalStore<TO>::put(pv[k]);
        if constexpr (COPY) qcopy[i] = ModalStore<TO>::put(qv[k]);
    }
}

// D (8x8) += A (8x4, row) B (4x8, col) in FP64.  Lane t holds A[t/4][t%4], B[t%4][t/4] and
// D[t/4][2 (t%4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// The contractions with the field as the A operand: its 8 rows are the real and imaginary parts of
// four neighbouring modes, so a warp reads and writes 64 contiguous bytes per layer; K and N run
// over the layers.  The first product's accumulator holds, in lane t, the modal amplitudes
// 2 (t%4) + {0, 1} of row t/4 -- which is the A operand of the second product if its K index is
// taken in the order (even modes, odd modes) of each group of eight.  The matrices are staged in
// that fragment order, one double per lane, so neither product needs a shuffle or a transpose.
// A warp takes two groups of four modes at a time, which halves the shared-memory reads of the
// fragments per product (one 256-byte read feeds two MMAs).
// Three CTAs per SM: 1, 2, 3, 4 of them took 189, 121.5, 107.9, 106.5 us for 16 layers on 2048^2
// and 35.5, 29.4, 29.5, 31.8 us for 32 on 512^2 (loads and MMAs of different warps overlap).  The
// floor of the latter is 14 us at the measured FP64 rate (4096 FMAs per mode), 9 us of traffic.
template <int NP, class TI, class TO, bool COPY>
__global__ void __launch_bounds__(256, 3) k_modal_mma(Geom g, const ModalConst* __restrict__ mc,
                                                      const TI* __restrict__ q, TO* __restrict__ psi,
                                                      TO* __restrict__ qcopy) {
    QGN_PDL_ENTRY();
    constexpr int KC = NP / 4, NT = NP / 8;
    using RI = decltype(TI::x);
    using RO = decltype(TO::x);
    extern __shared__ __align__(128) unsigned char sm_raw[];
    double* fp = reinterpret_cast<double*>(sm_raw);   // [KC][NT][32] proj fragments
    double* fb = fp + KC * NT * 32;                   // [NT][2][NT][32] back fragments
    const int nz = g.nz;
    for (int i = threadIdx.x; i < KC * NT * 32; i += blockDim.x) {
        const int t = i % 32, f = i / 32;
        {   // chunk c of four layers, tile n of eight modes
            const int c = f / NT, n = 8 * (f % NT) + t / 4, kk = 4 * c + t % 4;
            fp[i] = (n < nz && kk < nz) ? mc->proj[n * nz + kk] : 0.0;
        }
        {   // modes 8 tn + 2 (t%4) + par, tile u of eight layers
            const int tn = f / (2 * NT), par = (f / NT) % 2, u = f % NT;
            const int n = 8 * tn + 2 * (t % 4) + par, l = 8 * u + t / 4;
            fb[i] = (n < nz && l < nz) ? mc->back[l * nz + n] : 0.0;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x % 32;
    const int row = lane / 4, col = lane % 4;       // field row (2 mode + part), K or N index
    const int part = row & 1;
    double ev[NT];                                  // this lane's eigenvalue of each tile: its parity is its part
    const double Htot = mc->Htot;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int k = 8 * n + 2 * col + part;
        ev[n] = k < nz ? mc->evals[k] : -1.0;
    }
    const unsigned P = (unsigned)(g.nkx * g.nky), nky = (unsigned)g.nky;
    const unsigned warps = gridDim.x * (blockDim.x / 32);
    const unsigned w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    for (unsigned base = w * 8; base < P; base += warps * 8) {
        unsigned pm[2];                             // this lane's mode in each group
        bool ok[2];
        double a[2][KC];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            pm[h] = base + 4 * h + row / 2;
            ok[h] = pm[h] < P;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const int kk = 4 * c + col;
                const size_t i = (size_t)kk * P + pm[h];
                a[h][c] = 0.0;
                if (ok[h] && kk < nz && in_bounds(g, i, g.csize())) {
                    const RI v = reinterpret_cast<const RI*>(q)[2 * i + part];
                    a[h][c] = v;
                    if constexpr (COPY) reinterpret_cast<RO*>(qcopy)[2 * i + part] = (RO)v;
                }
            }
        }
        double m0[2][NT], m1[2][NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            m0[0][n] = m1[0][n] = m0[1][n] = m1[1][n] = 0.0;
#pragma unroll
            for (int c = 0; c < KC; ++c) {
                const double b = fp[(c * NT + n) * 32 + lane];
                mma_f64(m0[0][n], m1[0][n], a[0][c], b);
                mma_f64(m0[1][n], m1[1][n], a[1][c], b);
            }
        }
        // psi_mode = q_mode / ((-k^2 + EVals) Htot), zero for the mean mode.  The two rows of a
        // mode need the same two factors: each forms one and takes the other from its partner.
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const unsigned kx = pm[h] / nky, m = pm[h] % nky;
            const double kxv = g.dkx * (int)kx, kyv = g.kyval(g.jfull((int)m));
            const double k2 = kxv * kxv + kyv * kyv;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const double r = 1.0 / ((-k2 + ev[n]) * Htot);
                const double s = __shfl_xor_sync(0xffffffffu, r, 4);
                m0[h][n] = pm[h] == 0 ? 0.0 : m0[h][n] * (part ? s : r);
                m1[h][n] = pm[h] == 0 ? 0.0 : m1[h][n] * (part ? r : s);
            }
        }
#pragma unroll
        for (int u = 0; u < NT; ++u) {
            double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const double be = fb[((n * 2 + 0) * NT + u) * 32 + lane];
                const double bo = fb[((n * 2 + 1) * NT + u) * 32 + lane];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    mma_f64(d0[h], d1[h], m0[h][n], be);
                    mma_f64(d0[h], d1[h], m1[h][n], bo);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int l = 8 * u + 2 * col + i;
                    const size_t e = (size_t)l * P + pm[h];
                    if (ok[h] && l < nz && in_bounds(g, e, g.csize()))
                        reinterpret_cast<RO*>(psi)[2 * e + part] = (RO)(i ? d1[h] : d0[h]);
                }
            }
        }
    }
}

template <int NZ, class TI, class TO, bool COPY>
static void modal_small(const Geom& g, const Buffers& b, const TI* q, TO* psi, TO* qcopy, cudaStream_t s) {
    const unsigned grid = (unsigned)(((size_t)g.nkx * g.nky + 255) / 256);
    ::qgn::launch(k_modal<NZ, TI, TO, COPY>, grid, 256, 0, s, g, modal_params<NZ>(*b.mc_h), q, psi, qcopy);
}

template <int NP, class TI, class TO, bool COPY>
static void modal_wide(const Geom& g, const Buffers& b, const TI* q, TO* psi, TO* qcopy, cudaStream_t s) {
    const unsigned tiles = (unsigned)(((size_t)g.nkx * g.nky + 63) / 64);   // 8 warps of 8 modes per CTA
    const unsigned grid = tiles < 3 * 148 ? tiles : 3 * 148;
    constexpr int SMEM = 2 * (NP / 4) * (NP / 8) * 32 * (int)sizeof(double);
    ::qgn::launch(k_modal_mma<NP, TI, TO, COPY>, grid, 256, SMEM, s, g, b.mc, q, psi, qcopy);
}

template <class TI, class TO, bool COPY>
static cudaError_t launch_modal_any(const Geom& g, const Buffers& b, const TI* q, TO* psi, TO* qcopy, cudaStream_t s) {
    const double nb = (double)g.csize() * (sizeof(TI) + sizeof(TO) * (COPY ? 2.0 : 1.0));
    auto go = [&]() {
        switch (g.nz) {
            case 2: return modal_small<2, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 3: return modal_small<3, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 4: return modal_small<4, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 5: return modal_small<5, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 6: return modal_small<6, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 7: return modal_small<7, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            case 8: return modal_small<8, TI, TO, COPY>(g, b, q, psi, qcopy, s);
            default: break;
        }
        if constexpr (sizeof(TI) == 8)
            if (g.nz == 16) return modal_small<16, TI, TO, COPY>(g, b, q, psi, qcopy, s);
        if (g.nz <= 16) return modal_wide<16, TI, TO, COPY>(g, b, q, psi, qcopy, s);
        if (g.nz <= 24) return modal_wide<24, TI, TO, COPY>(g, b, q, psi, qcopy, s);
        return modal_wide<32, TI, TO, COPY>(g, b, q, psi, qcopy, s);
    };
    QGN_LAUNCH(KID_MODAL, nb, s, go());
    return cudaGetLastError();
}

cudaError_t launch_modal(const Geom& g, const Buffers& b, const double2* q, double2* psi, cudaStream_t s) {
    return launch_modal_any<double2, double2, false>(g, b, q, psi, nullptr, s);
}

// GetPsi of an FP32 field with FP64 arithmetic (mixed mode)
cudaError_t launch_modal_f32(const Geom& g, const Buffers& b, const float2* q, float2* psi, cudaStream_t s) {
    return launch_modal_any<float2, float2, false>(g, b, q, psi, nullptr, s);
}

// FP32 copy of the FP64 state and its GetPsi (FP64 arithmetic, FP32 result)
cudaError_t launch_modal_mixed(const Geom& g, const Buffers& b, const double2* q, float2* q32, float2* psi32,
                               cudaStream_t s) {
    return launch_modal_any<double2, float2, true>(g, b, q, psi32, q32, s);
}

}  // namespace qgn
