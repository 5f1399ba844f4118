// Fused DG tendency + LSRK stage kernels for brick meshes (sm_103a).
//
// One CTA owns one element for a whole stage:
//   phase 1  every node loads its state (coalesced), evaluates the dry
//            AtmosModel thermodynamics and its first-order flux in the three
//            directions and stages them in shared memory;
//   phase 2  every face node (6 (N+1)^2 of them) gathers the neighbour's
//            state at the matching node, forms the Rusanov (or central)
//            flux F*.n and stores it lifted, vMI*sM*F*, in shared memory
//            (without the interior half of its central part, which cancels
//            against the diagonal of the derivative: KParams::DhatC);
//   phase 3  every node contracts the staged fluxes with the weak-form
//            derivative Dhat = M^-1 D^T M along xi1, xi2, xi3, subtracts its
//            face terms, adds gravity and finishes either the tendency
//            T = alpha*dQ/dt + beta*T or the LSRK 2N stage update.  The
//            register holds the unscaled stage increment:
//            dq_s = dQ/dt(Q_{s-1}) + A_s dq_{s-1}, Q_s = Q_{s-1} + B_s dt dq_s,
//            which is the reference's dQ <- dQ/dt + dQ; Q <- Q + B_s dt dQ;
//            dQ <- A_{s+1} dQ with the A-scaling moved into the next stage
//            (one FMA per DOF; A_1 = 0, so stage 1 does not read the register
//            and stage 5 does not write it).
// The state is read from one buffer and the stage's new state written to
// another, so neighbouring elements never see a half-updated state.
//
// Algorithm restated from src/Numerics/DGMethods/DGModel_kernels.jl:64-548
// (volume_tendency!, H and V), :588-901 (dgsem_interface_tendency!),
// src/Numerics/DGMethods/NumericalFluxes.jl:219-340 (Rusanov / central),
// src/Atmos/Model/{tendencies_mass.jl:7-9, tendencies_momentum.jl:13-29,60-72,
// tendencies_energy.jl:7-21, AtmosModel.jl:776-796, bc_momentum.jl:25-34} and
// src/Numerics/ODESolvers/LowStorageRungeKuttaMethod.jl:102-158.
//
// On an affine brick element the contravariant flux M xi_d . F reduces to
// J w_i w_j w_k (2/dx_d) F_d, so the volume term at node (i,j,k) is
// (2/dx_1) sum_n Dhat[i][n] F_1(n,j,k) + ... with Dhat[i][n] = D[n][i] w_n / w_i,
// and the lift vMI*sM on a face normal to xi_d is (2/dx_d) / w_0.
//
// Precision: R = double (plain FP64) or R = float (mixed).  In the mixed
// form the state held in memory is the FP32 perturbation q' = q - q_ref about
// the FP64 hydrostatic reference state; pressure is formed directly as the
// perturbation p' = (R/cv)(rhoe' - |rhou|^2/(2 rho)) + rho' (R T0 - (R/cv) Phi),
// which is exact algebra for dry air (T = T0 + e_int/cv, p = rho R T), the
// reference-state jump across vertical faces enters the Rusanov penalty
// from an FP64-computed table, and the RK register dQ stays FP64.
//
// The FP64 form is bound by the FP64 pipe (1.8 lane operations per cycle and
// SM), so its operations are counted: reciprocals and roots of 3 and 5
// operations (rcp_r, sqrt_r), the metric folded into the derivative
// coefficients, no diagonal in the contraction, comparisons on the integer
// pipe.  A step of the 1 M-node bubble went from 2.304 to 1.665 ms (1.852 ms
// before the diagonal, and chained launches, launch.cuh).  In FP32 the same
// identity saves the face threads five loads and ten operations (0.167 to
// 0.164 ms).
#include <cooperative_groups.h>

#include "dg_common.cuh"

namespace cg = cooperative_groups;

namespace cmdg {
namespace {

template <int N>
struct Dims {
    static constexpr int Nq = N + 1;
    static constexpr int Nfp = Nq * Nq;
    static constexpr int Np = Nq * Nq * Nq;
    static constexpr int NF = 6 * Nfp;
    static constexpr int NT = (((Np > NF) ? Np : NF) + 31) / 32 * 32;
    // resident CTAs per SM requested for the FP32 kernels (register budget
    // 65536 / (NT * MIN_CTAS): 85, 85, 68 and 73 registers for N = 2..5)
#ifndef CMDG_MIN_CTAS_N4
#define CMDG_MIN_CTAS_N4 6
#endif
    static constexpr int MIN_CTAS = N == 2 ? 12 : N == 3 ? 8 : N == 4 ? CMDG_MIN_CTAS_N4 : 4;
    // the FP64 kernels are FP64-pipe bound; they keep enough CTAs to cover the barriers
    static constexpr int MIN_CTAS64 = N == 5 ? 2 : 3;
    // one CTA per element (no look-ahead registers): a tighter register budget
#ifndef CMDG_MIN_CTAS_DIRECT_N4
#define CMDG_MIN_CTAS_DIRECT_N4 7
#endif
    static constexpr int MIN_CTAS_DIRECT = N == 2 ? 16 : N == 3 ? 12 : N == 4 ? CMDG_MIN_CTAS_DIRECT_N4 : 5;
};

template <int N, typename R>
struct Smem {
    static constexpr int Nq = N + 1, Np = Nq * Nq * Nq, Nfp = Nq * Nq;
    // planar five-field records (Planar5): node states and volume fluxes by
    // direction; (sound speed, 1/rho) pairs per node; the lifted face fluxes
    // in node-major scalar planes, one set per face direction (a node lies
    // on at most one face of each direction), so a node reads its face terms
    // with consecutive 4- or 8-byte accesses
    static constexpr int P5N = planar_pad<R>(5 * Np);      // one five-field plane set over the nodes
    static constexpr int NODE = 0;
    static constexpr int CR = NODE + P5N;
    static constexpr int FLUX = CR + planar_pad<R>(2 * Np);
    static constexpr int FACE = FLUX + 3 * P5N;
    static constexpr int DMAT = FACE + planar_pad<R>(3 * 5 * Np);
    // FP64: the derivative already scaled by the metric, one copy per direction
    static constexpr int TOTAL = DMAT + (sizeof(R) == 8 ? 3 : 1) * Nq * Nq;
    static constexpr size_t BYTES = sizeof(R) * TOTAL;
};

// Double-buffered staging of the persistent kernel (byte offsets after
// Smem): per buffer the 16-byte-aligned window around one element's state
// block (5 x Np words of R; the element's block starts 0..15 bytes into the
// window) and around its RK register block (5 x Np doubles), then one
// mbarrier per buffer.
template <int N, typename R>
struct SmemTma {
    static constexpr int Np = (N + 1) * (N + 1) * (N + 1);
    static constexpr size_t QB = (Smem<N, R>::BYTES + 15) / 16 * 16;
    static constexpr size_t QBLK = (NSTATE * Np * sizeof(R) + 32 + 15) / 16 * 16;
    static constexpr size_t DB = QB + 2 * QBLK;
    static constexpr size_t DBLK = (NSTATE * Np * sizeof(double) + 32 + 15) / 16 * 16;
    static constexpr size_t BAR = DB + 2 * DBLK;
    static constexpr size_t BYTES = BAR + 2 * sizeof(uint64_t);
};

// 16-byte-aligned window [lo, hi) around the byte range [a, a + n) of an
// array [base, end); false when the window leaves the array (then the
// element is read with plain loads).
__device__ __forceinline__ bool bulk_window(uintptr_t base, uintptr_t end, uintptr_t a, size_t n, uintptr_t& lo,
                                            uint32_t& bytes) {
    lo = a & ~(uintptr_t)15;
    const uintptr_t hi = (a + n + 15) & ~(uintptr_t)15;
    bytes = (uint32_t)(hi - lo);
    return lo >= base && hi <= end;
}

// Per-element inputs of one thread.
template <typename R>
struct Ahead {
    R q[NSTATE];   // own node state (node threads)
    R qp[NSTATE];  // neighbour state at this thread's face node (face threads)
    int nb;        // neighbour element across this thread's face, or -tag
    int ez;        // vertical element index of the element
};

// Processes elements e_first, e_first + e_stride, ... below e_end with the
// whole CTA.  PERSIST: a grid of resident CTAs walks the elements; while it
// computes one element, the TMA engine copies the next element's state and
// RK register blocks (contiguous in the (Np, 5, nelem) layout) into the other
// of two shared-memory buffers, so every CTA keeps memory requests in flight
// throughout without per-thread copy instructions.
// PARAM_D: the weak-form derivative is read from the kernel parameter's
// constant bank (a constant-cache load with the thread's row index) instead
// of a shared-memory copy.  The one-model kernels keep the shared copy: on
// the 1 M-node bubble it measured 0.1828 ms per mixed step against 0.1846 ms
// from the constant bank, whose reads differ in address across a warp; the
// cluster kernel reads the constant bank.
template <typename R>
__device__ __forceinline__ R dhat_const(const KParams& P, int idx);
template <>
__device__ __forceinline__ float dhat_const<float>(const KParams& P, int idx) {
    return P.DhatC32[idx];
}
template <>
__device__ __forceinline__ double dhat_const<double>(const KParams& P, int idx) {
    return P.DhatC64[idx];
}

template <int N, typename R, bool MIXED, int MODE, bool PERSIST, bool PARAM_D, int CL = 0>
__device__ __forceinline__ void stage_body(const KParams& P, unsigned char* smem_raw, int e_first, int e_stride,
                                           int e_end, int release) {
    static_assert(CL == 0 || CL == 2 || CL == 4 || CL == 8, "clusters of 2 (z), 4 (x, z) or 8 (x, y, z) elements");
    static_assert(CL == 0 || !PERSIST, "a cluster CTA computes one element");
    using Dm = Dims<N>;
    using SM = Smem<N, R>;
    constexpr int Nq = Dm::Nq, Np = Dm::Np, Nfp = Dm::Nfp;
    constexpr int ESTRIDE = NSTATE * Np;  // elements of R (or double) per element
    using PL = Planar5<R>;
    using CRV = typename Pair<R>::V;
    R* const sm = reinterpret_cast<R*>(smem_raw);
    R* const s_node = sm + SM::NODE;
    CRV* const s_cr = reinterpret_cast<CRV*>(sm + SM::CR);
    R* const s_F = sm + SM::FLUX;
    R* const s_fs = sm + SM::FACE;
    R* const s_D = sm + SM::DMAT;

    const int t = threadIdx.x;
    const R* Qin = static_cast<const R*>(P.Qin);
    R* Qout = static_cast<R*>(P.Qout);
    const Physics& ph = P.ph;
    const bool node_thread = t < Np;
    const bool face_thread = t < 6 * Nfp;
    const bool read_reg = (MODE == 0) ? (P.beta != 0) : !P.first_stage;

    // ---------------- element-independent per-thread geometry
    // node thread: (i, j, k) and its three contraction lines
    const int nk = node_thread ? t / Nfp : 0;
    const int nj = node_thread ? (t - nk * Nfp) / Nq : 0;
    const int ni = node_thread ? t - nk * Nfp - nj * Nq : 0;
    // face thread: face f (0..5 = xi1-, xi1+, xi2-, xi2+, xi3-, xi3+), in-face node fn.
    // CL: the CTA's rank in its cluster of 2 x 2 x 2 (CL = 8), 2 x 1 x 2 (4)
    // or 1 x 1 x 2 (2) elements, bit 0 = upper in z, bit 1 = upper in x,
    // bit 2 = upper in y.  The faces shared with the other elements of the
    // cluster take the first face slots, so whole warps read their neighbour
    // from that element's shared memory and the rest gather it from global
    // memory (a warp that mixes the two paths runs both).
    const int crank = CL > 0 ? (int)(blockIdx.x % (unsigned)(CL > 0 ? CL : 1)) : 0;
    constexpr int NIN = CL == 8 ? 3 : (CL == 4 ? 2 : (CL == 2 ? 1 : 0));  // dimensions the cluster spans
    // slot -> face: slots 0 .. NIN-1 the faces towards the other half of the
    // cluster in z, x, y (bit b of the rank: upper half -> the minus face);
    // NIN .. 2 NIN - 1 the opposite faces; then both faces of each direction
    // the cluster does not span
    auto slot_face = [&](int slot) {
        auto dir = [](int dim) { return dim == 0 ? 2 : (dim == 1 ? 0 : 1); };  // cluster dimension z, x, y
        if (slot < 2 * NIN) {
            const int dim = slot < NIN ? slot : slot - NIN;
            const int upper = (crank >> dim) & 1;
            const int side = (slot < NIN) ? (upper ^ 1) : upper;
            return 2 * dir(dim) + side;
        }
        const int rest = slot - 2 * NIN;
        return 2 * dir(NIN + rest / 2) + (rest & 1);
    };
    const int fslot = face_thread ? t / Nfp : 0;
    const int f = CL > 0 ? slot_face(fslot) : fslot;
    const bool remote = CL > 0 && face_thread && fslot < NIN;  // neighbour inside the cluster
    const int nrank = remote ? (crank ^ (1 << fslot)) : 0;
    const int fn = face_thread ? t - fslot * Nfp : 0;
    const int fd = f >> 1, fside = f & 1;
    const int fa = fn % Nq, fb = fn / Nq;
    // volume node on face f at in-face (a, b), and the matching node of the neighbour on face f^1
    const int vM = fd == 0 ? fside * N + Nq * fn : (fd == 1 ? fa + Nq * (fside * N + Nq * fb) : fn + Nfp * (fside * N));
    const int oside = fside ^ 1;
    const int vP = fd == 0 ? oside * N + Nq * fn : (fd == 1 ? fa + Nq * (oside * N + Nq * fb) : fn + Nfp * (oside * N));
    const int kM = vM / Nfp, kP = vP / Nfp;
    // record of this node in the plane of the direction-d flux: the
    // contraction index d is the slowest (d = 2 is the natural order), so a
    // warp reading one position n of many lines, or one face, touches
    // consecutive records
    auto dir_rec = [&](int d) {
        return d == 0 ? ni * Nfp + (nj + Nq * nk) : (d == 1 ? nj * Nfp + (ni + Nq * nk) : t);
    };
    const R sgn = fside ? R(1) : R(-1);

    // FP64: the element's metric goes into the derivative coefficients (three
    // copies, one multiplication per coefficient of the element instead of
    // three per node and field)
    constexpr bool SCALED_D = sizeof(R) == 8;
    if (!PARAM_D && !SCALED_D && t < Nq * Nq) s_D[t] = static_cast<const R*>(P.Dhat)[t];

    auto fetch = [&](int e, Ahead<R>& a) {
        const int* nbr = P.nbr + NBR_STRIDE * e;
        a.ez = __ldg(nbr + 6);
        a.nb = face_thread ? __ldg(nbr + f) : -1;
        chain_wait();
        if (node_thread) {
            const R* qe = Qin + (size_t)e * ESTRIDE + t;
#pragma unroll
            for (int s = 0; s < NSTATE; ++s) a.q[s] = qe[s * Np];
        }
        if (a.nb >= 0 && !remote) {
            const R* qn = Qin + (size_t)a.nb * ESTRIDE + vP;
#pragma unroll
            for (int s = 0; s < NSTATE; ++s) a.qp[s] = qn[s * Np];
        }
    };

    // persistent staging: buffers, barriers, and the copy issue by thread 0
    using ST = SmemTma<N, R>;
    uint64_t* const bars = reinterpret_cast<uint64_t*>(smem_raw + ST::BAR);
    const uintptr_t q_base = reinterpret_cast<uintptr_t>(Qin);
    const uintptr_t q_end = q_base + (size_t)P.nelem * ESTRIDE * sizeof(R);
    const uintptr_t d_base = reinterpret_cast<uintptr_t>(P.dQ);
    const uintptr_t d_end = d_base + (size_t)P.nelem * ESTRIDE * sizeof(double);
    // window of element ee's state (fs) and register (fd) blocks; shifts in words
    auto windows = [&](int ee, uintptr_t& qlo, uint32_t& qbytes, bool& qok, uintptr_t& dlo, uint32_t& dbytes,
                       bool& dok) {
        const uintptr_t qa = q_base + (size_t)ee * ESTRIDE * sizeof(R);
        qok = bulk_window(q_base, q_end, qa, ESTRIDE * sizeof(R), qlo, qbytes);
        dok = false;
        dbytes = 0;
        dlo = 0;
        if (read_reg) {
            const uintptr_t da = d_base + (size_t)ee * ESTRIDE * sizeof(double);
            dok = bulk_window(d_base, d_end, da, ESTRIDE * sizeof(double), dlo, dbytes);
        }
    };
    int issued0 = 0, issued1 = 0;  // copies armed per buffer (thread 0)
    auto issue = [&](int ee, int b) {  // thread 0 only
        if (b) ++issued1;
        else ++issued0;
        uint32_t total = 0;
        uintptr_t qlo = 0, dlo = 0;
        uint32_t qbytes = 0, dbytes = 0;
        bool qok = false, dok = false;
        if (ee < e_end) {
            windows(ee, qlo, qbytes, qok, dlo, dbytes, dok);
            total = (qok ? qbytes : 0u) + (dok ? dbytes : 0u);
        }
        if (P.staging_skip_copies) qok = dok = false;  // test hook: the armed bytes never arrive
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bars[b], total);
        if (qok) bulk_copy_g2s(smem_raw + ST::QB + b * ST::QBLK, reinterpret_cast<const void*>(qlo), qbytes, &bars[b]);
        if (dok) bulk_copy_g2s(smem_raw + ST::DB + b * ST::DBLK, reinterpret_cast<const void*>(dlo), dbytes, &bars[b]);
    };
    bool timed_out = false;

    int e = e_first;
    Ahead<R> cur;
    if (PERSIST) {
        chain_wait();
        if (t == 0) {
            mbar_init(&bars[0], 1);
            mbar_init(&bars[1], 1);
            mbar_fence_init();
        }
        __syncthreads();
        if (t == 0) issue(e, 0);
    }
    for (int it = 0; e < e_end; e += e_stride, ++it) {
        const int b = it & 1;
        double dq_old[NSTATE];
        const size_t ebase = (size_t)e * ESTRIDE + t;
        if (PERSIST) {
            // the other buffer was read at the start of the previous element,
            // before that element's closing barrier: copy the next element into it
            if (t == 0) issue(e + e_stride, b ^ 1);
            const int* nbr = P.nbr + NBR_STRIDE * e;
            cur.ez = __ldg(nbr + 6);
            cur.nb = face_thread ? __ldg(nbr + f) : -1;
            if (cur.nb >= 0) {
                const R* qn = Qin + (size_t)cur.nb * ESTRIDE + vP;
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) cur.qp[s] = qn[s * Np];
            }
            const bool arrived = mbar_wait_bounded(&bars[b], (uint32_t)((it >> 1) & 1), P.wait_polls);
            // a staging copy that did not complete in time: every thread of
            // the CTA stops here, before an element is computed from the
            // unfilled buffer and before a barrier whose phase is still open
            // would be armed again (one arrival per phase)
            if (__syncthreads_or(!arrived)) {
                timed_out = true;
                break;
            }
            uintptr_t qlo, dlo;
            uint32_t qbytes, dbytes;
            bool qok, dok;
            windows(e, qlo, qbytes, qok, dlo, dbytes, dok);
            if (node_thread) {
                if (qok) {
                    const R* qs = reinterpret_cast<const R*>(smem_raw + ST::QB + b * ST::QBLK) +
                                  (q_base + (size_t)e * ESTRIDE * sizeof(R) - qlo) / sizeof(R);
#pragma unroll
                    for (int s = 0; s < NSTATE; ++s) cur.q[s] = qs[s * Np + t];
                } else {
#pragma unroll
                    for (int s = 0; s < NSTATE; ++s) cur.q[s] = Qin[ebase + s * Np];
                }
                if (read_reg) {
                    if (dok) {
                        const double* ds = reinterpret_cast<const double*>(smem_raw + ST::DB + b * ST::DBLK) +
                                           (d_base + (size_t)e * ESTRIDE * sizeof(double) - dlo) / sizeof(double);
#pragma unroll
                        for (int s = 0; s < NSTATE; ++s) dq_old[s] = ds[s * Np + t];
                    } else {
#pragma unroll
                        for (int s = 0; s < NSTATE; ++s) dq_old[s] = P.dQ[ebase + s * Np];
                    }
                }
            }
        } else {
            fetch(e, cur);
            if (node_thread && read_reg) {
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) dq_old[s] = P.dQ[ebase + s * Np];
            }
        }

        const int ez = cur.ez;
        const R xi[3] = {KConst<R>::metric(P, e, 0), KConst<R>::metric(P, e, 1), KConst<R>::metric(P, e, 2)};

        if (SCALED_D && t < Nq * Nq) {
            const R d = static_cast<const R*>(P.Dhat)[t];
#pragma unroll
            for (int dd = 0; dd < 3; ++dd) s_D[dd * Nq * Nq + t] = d * xi[dd];
        }

        // ---------------- phase 1: node thermodynamics and volume fluxes
        R gsrc = 0;
        if (node_thread) {
            const Level<R> lv = load_level<R>(P, ez * Nq + nk);
            const Thermo<R, MIXED> th = thermo<R, MIXED>(cur.q, lv, P);
            PL::st(s_node, Np, t, cur.q);
            s_cr[t] = Pair<R>::make(th.c, th.rinv);
#pragma unroll
            for (int dd = 0; dd < 3; ++dd) {
                R F[NSTATE];
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) F[s] = flux_d<R, MIXED>(cur.q, th, dd, s);
                PL::st(s_F + dd * SM::P5N, Np, dir_rec(dd), F);
            }
            if (ph.gravity) {
                R rho_s = MIXED ? ((ph.ref_state && ph.subtract_off) ? cur.q[0] : lv.rho_ref + cur.q[0])
                                : ((ph.ref_state && ph.subtract_off) ? cur.q[0] - lv.rho_ref : cur.q[0]);
                gsrc = -rho_s * lv.gphiz;
            }
        }
        // CL: every element of the cluster has staged its nodes before any reads them
        if constexpr (CL > 0) cg::this_cluster().sync();
        else __syncthreads();

        // ---------------- phase 2: one numerical flux per face node
        if (face_thread) {
            R qm[NSTATE], Fp[NSTATE], qp[NSTATE], jr[NSTATE] = {0, 0, 0, 0, 0};
            PL::ld(s_node, Np, vM, qm);
            const CRV cr = s_cr[vM];
            const R c_m = cr.x, ri_m = cr.y;
            const R lam_m = fabs(pick3(fd, qm[1], qm[2], qm[3]) * ri_m) + c_m;
            int ezp = ez;
            if (cur.nb >= 0) {
                if (!remote) {
#pragma unroll
                    for (int s = 0; s < NSTATE; ++s) qp[s] = cur.qp[s];
                }
                if (fd == 2) {
                    // vertical neighbour: one element below (f = 4) or above (f = 5), periodic wrap
                    ezp = ez + (fside ? 1 : -1);
                    ezp = ezp < 0 ? ezp + P.nz : (ezp >= P.nz ? ezp - P.nz : ezp);
                    if (MIXED && ph.numflux == CMDG_FLUX_RUSANOV) {
                        // reference-state jump q_ref(-) - q_ref(+) across the face
                        const int ej = fside ? ezp : ez;
                        const R sj = fside ? R(-1) : R(1);
                        jr[0] = sj * (R)P.jump32[2 * ej + 0];
                        jr[4] = sj * (R)P.jump32[2 * ej + 1];
                    }
                }
            } else {
                // Impenetrable(FreeSlip) + Insulating wall: rhou+ = rhou- - 2 (rhou-.n) n
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) qp[s] = qm[s];
                qp[1] = (fd == 0) ? -qm[1] : qm[1];
                qp[2] = (fd == 1) ? -qm[2] : qm[2];
                qp[3] = (fd == 2) ? -qm[3] : qm[3];
            }
            R lam_p;
            if (CL > 0 && remote) {
                // the neighbour inside the cluster: its staged state, (c, 1/rho)
                // and xi_fd flux at the facing node, read from its shared memory
                const auto cl = cg::this_cluster();
                PL::ld(cl.map_shared_rank(s_node, (unsigned)nrank), Np, vP, qp);
                const CRV crp = cl.map_shared_rank(s_cr, (unsigned)nrank)[vP];
                PL::ld(cl.map_shared_rank(s_F + fd * SM::P5N, (unsigned)nrank), Np, oside * N * Nfp + fn, Fp);
                lam_p = fabs(pick3(fd, qp[1], qp[2], qp[3]) * crp.y) + crp.x;
            } else {
                const Level<R> lvp = load_level<R>(P, ezp * Nq + (cur.nb >= 0 ? kP : kM));
                const Thermo<R, MIXED> thp = thermo<R, MIXED, MIXED>(qp, lvp, P);
                if (MIXED) {
                    normal_flux<R, MIXED>(qp, thp, fd, R(1), Fp);
                    lam_p = fabs(pick3(fd, thp.u[0], thp.u[1], thp.u[2])) + thp.c;
                } else {
                    const R mn = pick3(fd, qp[1], qp[2], qp[3]);
                    const R un = mn * thp.rinv;
                    far_flux_d<R>(qp, mn, un, thp.pflux, thp.H, fd, Fp);
                    lam_p = fabs(un) + thp.c;
                }
            }
            // the central part's interior half is left out with the diagonal
            // of the derivative (KParams::DhatC)
            const R lift = pick3(fd, xi[0], xi[1], xi[2]) * KConst<R>::inv_w0(P);
            const R hmw = (ph.numflux == CMDG_FLUX_RUSANOV) ? R(0.5) * max_nonneg(lam_m, lam_p) : R(0);
            const R hl = (R(0.5) * sgn) * lift, pl = hmw * lift;
            R fs[NSTATE];
            if (MIXED) {
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) fs[s] = hl * Fp[s] + pl * ((qm[s] - qp[s]) + jr[s]);
            } else {
                lifted_flux<R, MIXED>(Fp, qm, qp, R(0), R(0), hl, pl, fs);
            }
#pragma unroll
            for (int s = 0; s < NSTATE; ++s) s_fs[(fd * NSTATE + s) * Np + vM] = fs[s];
        }
        // CL: no element of the cluster leaves (or reuses its shared memory)
        // while another may still read it
        if constexpr (CL > 0) cg::this_cluster().sync();
        else __syncthreads();

        if (release) chain_release();

        // ---------------- phase 3: volume contraction, face terms, source, update
        int bad = 0;
        if (node_thread) {
            R rhs[NSTATE];
            const int L1 = nj + Nq * nk;  // line along xi1 (records n Nfp + L1)
            const int L2 = ni + Nq * nk;  // line along xi2 (records n Nfp + L2)
            const int L3 = ni + Nq * nj;         // line along xi3 (stride Nfp)
            R acc1[NSTATE] = {0, 0, 0, 0, 0}, acc2[NSTATE] = {0, 0, 0, 0, 0}, acc3[NSTATE] = {0, 0, 0, 0, 0};
#pragma unroll
            for (int n = 0; n < (SCALED_D ? N : Nq); ++n) {
                const int n1 = SCALED_D ? others(n, ni) : n, n2 = SCALED_D ? others(n, nj) : n,
                          n3 = SCALED_D ? others(n, nk) : n;
                R v1[NSTATE], v2[NSTATE], v3[NSTATE];
                PL::ld(s_F, Np, L1 + n1 * Nfp, v1);
                PL::ld(s_F + SM::P5N, Np, L2 + n2 * Nfp, v2);
                PL::ld(s_F + 2 * SM::P5N, Np, L3 + n3 * Nfp, v3);
                if constexpr (SCALED_D) {
                    const R d1 = s_D[ni * Nq + n1], d2 = s_D[Nq * Nq + nj * Nq + n2],
                            d3 = s_D[2 * Nq * Nq + nk * Nq + n3];
#pragma unroll
                    for (int s = 0; s < NSTATE; ++s) {
                        acc1[s] = fma(d1, v1[s], acc1[s]);
                        acc1[s] = fma(d2, v2[s], acc1[s]);
                        acc1[s] = fma(d3, v3[s], acc1[s]);
                    }
                } else {
                    const R d1 = PARAM_D ? dhat_const<R>(P, ni * Nq + n) : s_D[ni * Nq + n];
                    const R d2 = PARAM_D ? dhat_const<R>(P, nj * Nq + n) : s_D[nj * Nq + n];
                    const R d3 = PARAM_D ? dhat_const<R>(P, nk * Nq + n) : s_D[nk * Nq + n];
#pragma unroll
                    for (int s = 0; s < NSTATE; ++s) {
                        acc1[s] = fma(d1, v1[s], acc1[s]);
                        acc2[s] = fma(d2, v2[s], acc2[s]);
                        acc3[s] = fma(d3, v3[s], acc3[s]);
                    }
                }
            }
#pragma unroll
            for (int s = 0; s < NSTATE; ++s)
                rhs[s] = SCALED_D ? acc1[s] : xi[0] * acc1[s] + xi[1] * acc2[s] + xi[2] * acc3[s];
            // face terms (vMI sM F*, lifted in phase 2), in face order 1..6:
            // at most one face per direction holds the node
            auto sub_face = [&](int dd) {
#pragma unroll
                for (int s = 0; s < NSTATE; ++s) rhs[s] -= s_fs[(dd * NSTATE + s) * Np + t];
            };
            if (ni == 0 || ni == N) sub_face(0);
            if (nj == 0 || nj == N) sub_face(1);
            if (nk == 0 || nk == N) sub_face(2);
            rhs[3] += gsrc;
            const R rkb_dt = KConst<R>::rkb_dt(P);
#pragma unroll
            for (int s = 0; s < NSTATE; ++s) {
                if (!finite_r(rhs[s])) bad = 1;
                const size_t idx = ebase + s * Np;
                if (MODE == 0) {
                    double out = P.alpha * (double)rhs[s];
                    if (read_reg) out = fma(P.beta, dq_old[s], out);
                    P.dQ[idx] = out;
                } else {
                    // unscaled 2N register: dq_s = rhs_s + A_s dq_{s-1}  (A_1 = 0)
                    double dq;
                    if (MIXED) {
                        // one FP64 FMA per DOF; the conversions run on the integer pipe
                        if (read_reg) {
                            dq = fma(P.rka, dq_old[s], f32_to_f64_bits((float)rhs[s]));
                            Qout[idx] = fma(rkb_dt, (R)f64_to_f32_bits(dq), cur.q[s]);
                        } else {
                            dq = f32_to_f64_bits((float)rhs[s]);
                            Qout[idx] = fma(rkb_dt, rhs[s], cur.q[s]);
                        }
                    } else {
                        dq = read_reg ? fma(P.rka, dq_old[s], (double)rhs[s]) : (double)rhs[s];
                        Qout[idx] = (R)fma(P.rkb_dt, dq, (double)cur.q[s]);
                    }
                    if (!P.last_stage) P.dQ[idx] = dq;
                }
            }
        }
        if (PERSIST || e + e_stride < e_end) {
            // also separates this element's shared-memory reads from the next one's writes
            if (__syncthreads_or(bad) && t == 0) atomicOr(P.status, 1u);
        } else {
            // last element of this CTA: no barrier, one vote per warp
            if (__any_sync(0xffffffffu, bad) && (t & 31) == 0) atomicOr(P.status, 1u);
        }
    }
    if (PERSIST && timed_out) {
        // a staging copy did not complete in time: report it, and before the
        // CTA's shared memory is released wait (bounded) once more for the
        // copies of both buffers
        if (t == 0) {
            atomicOr(P.status, 2u);
            // phases complete in order: waiting for each buffer's latest armed phase covers the rest
            if (issued0 > 0) mbar_wait_bounded(&bars[0], (uint32_t)((issued0 - 1) & 1), P.wait_polls);
            if (issued1 > 0) mbar_wait_bounded(&bars[1], (uint32_t)((issued1 - 1) & 1), P.wait_polls);
        }
    }
}

template <int N, typename R, bool MIXED, int MODE, bool PERSIST, bool BACK = false>
__global__ void __launch_bounds__(Dims<N>::NT, MIXED ? (PERSIST ? Dims<N>::MIN_CTAS : Dims<N>::MIN_CTAS_DIRECT)
                                                     : Dims<N>::MIN_CTAS64) stage_kernel(const KParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if constexpr (PERSIST) {
        stage_body<N, R, MIXED, MODE, true, false>(P, smem_raw, blockIdx.x, gridDim.x, P.nelem,
                                                   P.release & RELEASE_STAGE);
    } else {
        const int e = element_of<BACK>();
        stage_body<N, R, MIXED, MODE, false, false>(P, smem_raw, e, 1, e + 1, P.release & RELEASE_STAGE);
    }
}

// One CTA per element in clusters of CL CTAs that are adjacent elements
// (2 x 2 x 2, 2 x 1 x 2 or 1 x 1 x 2 in x, y, z): the CTA of cluster rank r
// computes element P.cl_elem[blockIdx.x], and the faces shared inside the
// cluster read the neighbour's staged state and flux from its CTA's shared
// memory (distributed shared memory) instead of gathering the neighbour's
// state from global memory and recomputing its thermodynamics and flux.
template <int N, typename R, bool MIXED, int MODE, int CL>
__global__ void __launch_bounds__(Dims<N>::NT, MIXED ? Dims<N>::MIN_CTAS_DIRECT : Dims<N>::MIN_CTAS64)
    stage_cluster_kernel(const KParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int e = __ldg(P.cl_elem + blockIdx.x);
    stage_body<N, R, MIXED, MODE, false, true, CL>(P, smem_raw, e, 1, e + 1, P.release & RELEASE_STAGE);
}

template <int N, typename R, bool MIXED, int MODE, int CL>
cudaError_t launch_cluster_mode(const KParams& P, cudaStream_t s) {
    constexpr size_t bytes = Smem<N, R>::BYTES;
    static unsigned long long configured = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (bytes > 48 * 1024 && !(configured & (1ull << (dev & 63)))) {
        e = cudaFuncSetAttribute(stage_cluster_kernel<N, R, MIXED, MODE, CL>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        configured |= 1ull << (dev & 63);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P.nelem, 1, 1);
    cfg.blockDim = dim3(Dims<N>::NT, 1, 1);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, stage_cluster_kernel<N, R, MIXED, MODE, CL>, P);
}

template <int N, typename R, bool MIXED, int CL>
cudaError_t launch_cluster_typed(const KParams& P, int mode, cudaStream_t s) {
    return mode == 0 ? launch_cluster_mode<N, R, MIXED, 0, CL>(P, s) : launch_cluster_mode<N, R, MIXED, 1, CL>(P, s);
}

template <int N>
cudaError_t launch_cluster_N(const KParams& P, bool mixed, int mode, int cl, cudaStream_t s) {
    if (cl == 8)
        return mixed ? launch_cluster_typed<N, float, true, 8>(P, mode, s)
                     : launch_cluster_typed<N, double, false, 8>(P, mode, s);
    if (cl == 4)
        return mixed ? launch_cluster_typed<N, float, true, 4>(P, mode, s)
                     : launch_cluster_typed<N, double, false, 4>(P, mode, s);
    return mixed ? launch_cluster_typed<N, float, true, 2>(P, mode, s)
                 : launch_cluster_typed<N, double, false, 2>(P, mode, s);
}

template <int N, typename R, bool MIXED, int MODE, bool PERSIST, bool BACK = false>
cudaError_t launch_mode(const KParams& P, int grid_ctas, cudaStream_t s) {
    constexpr size_t bytes = PERSIST ? SmemTma<N, R>::BYTES : Smem<N, R>::BYTES;
    // per-device set-up: opt in to > 48 KB of dynamic shared memory and size a
    // persistent grid from the occupancy of this instantiation
    static int resident[64] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    dev &= 63;
    if (resident[dev] == 0) {
        if (bytes > 48 * 1024) {
            e = cudaFuncSetAttribute(stage_kernel<N, R, MIXED, MODE, PERSIST, BACK>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e != cudaSuccess) return e;
        }
        int per_sm = 0, sms = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stage_kernel<N, R, MIXED, MODE, PERSIST, BACK>,
                                                          Dims<N>::NT, bytes);
        if (e != cudaSuccess) return e;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        resident[dev] = (per_sm > 0 ? per_sm : 1) * sms;
    }
    int grid = PERSIST ? (grid_ctas > 0 ? grid_ctas : resident[dev]) : P.nelem;
    if (grid > P.nelem) grid = P.nelem;
    return launch_chained(s, stage_kernel<N, R, MIXED, MODE, PERSIST, BACK>, (unsigned)grid, Dims<N>::NT, bytes, P);
}

template <int N, typename R, bool MIXED>
cudaError_t launch_typed(const KParams& P, int mode, int grid, cudaStream_t s) {
    // grid < 0 selects one CTA per element; otherwise the persistent kernel
    if (grid < 0)
        return mode == 0    ? launch_mode<N, R, MIXED, 0, false>(P, 0, s)
               : P.backward ? launch_mode<N, R, MIXED, 1, false, true>(P, 0, s)
                            : launch_mode<N, R, MIXED, 1, false>(P, 0, s);
    return mode == 0 ? launch_mode<N, R, MIXED, 0, true>(P, grid, s) : launch_mode<N, R, MIXED, 1, true>(P, grid, s);
}

template <int N>
cudaError_t launch_N(const KParams& P, bool mixed, int mode, int grid, cudaStream_t s) {
    return mixed ? launch_typed<N, float, true>(P, mode, grid, s) : launch_typed<N, double, false>(P, mode, grid, s);
}

// ---------------------------------------------------------------------------
// Ensembles: one launch per stage and polynomial order advances every member
// of that order.  The CTAs walk a list of tiles (runs of consecutive elements
// of one member); each tile reads its member's launch parameters from global
// memory and runs the node-kernel body with the CTA shape of its order.
// Resident CTAs per SM: the persistent kernel's budget, except at N = 4,
// where reading each tile's launch parameters from global memory costs
// registers: 5 CTAs (72 registers, 20 bytes of spills) measured 1.203e11
// DOF-stage/s on the 64-member ensemble against 1.159e11 at 6 (64
// registers, 44 bytes of spills) and 1.17-1.19e11 at 4 (96, none).
template <int N>
constexpr int batch_min_ctas() {
    return N == 4 ? 5 : Dims<N>::MIN_CTAS;
}

template <int N>
__global__ void __launch_bounds__(Dims<N>::NT, batch_min_ctas<N>())
    batch_stage_kernel(const KParams* __restrict__ params, const BatchTile* __restrict__ tiles, int ntiles,
                       int release) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    chain_wait();
    for (int it = blockIdx.x; it < ntiles; it += gridDim.x) {
        const BatchTile T = tiles[it];
        stage_body<N, float, true, 1, false, false>(params[T.member], smem_raw, T.e0, 1, T.e1, release);
    }
}

template <int N>
cudaError_t launch_batch_N(const KParams* d_params, const BatchTile* d_tiles, int ntiles, int grid, cudaStream_t s) {
    constexpr size_t bytes = Smem<N, float>::BYTES;
    static unsigned long long configured = 0;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!(configured & (1ull << (dev & 63)))) {
        e = cudaFuncSetAttribute(batch_stage_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        configured |= 1ull << (dev & 63);
    }
    return launch_chained(s, batch_stage_kernel<N>, (unsigned)grid, Dims<N>::NT, bytes, d_params, d_tiles, ntiles,
                          chain_releases(grid, chain_ctas<batch_stage_kernel<N>>(Dims<N>::NT, bytes, dev)));
}

template <int N>
int stage_ctas_N(bool mixed) {
    return mixed ? chain_ctas<stage_kernel<N, float, true, 1, false, false>>(Dims<N>::NT, Smem<N, float>::BYTES)
                 : chain_ctas<stage_kernel<N, double, false, 1, false, false>>(Dims<N>::NT, Smem<N, double>::BYTES);
}

template <int N>
int resident_N() {
    int dev = 0, per_sm = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    constexpr size_t bytes = Smem<N, float>::BYTES;
    cudaFuncSetAttribute(batch_stage_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_stage_kernel<N>, Dims<N>::NT, bytes) !=
        cudaSuccess)
        return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return per_sm * sms;
}

}  // namespace

static int brick_stage_ctas(const Model* md) {
    const bool mixed = md->precision == CMDG_MIXED;
    switch (md->mesh->N) {
        case 2: return stage_ctas_N<2>(mixed);
        case 3: return stage_ctas_N<3>(mixed);
        case 4: return stage_ctas_N<4>(mixed);
        case 5: return stage_ctas_N<5>(mixed);
        default: return 0;
    }
}

int chain_flags(Model* md) {
    const int known = md->release.load(std::memory_order_relaxed);
    if (known >= 0) return known;
    const bool hyper = md->prm.hyperdiffusion != CMDG_HYPER_NONE, visc = md->prm.turbulence != CMDG_TURB_NONE;
    const int kind = md->mesh->kind;
    auto ctas = [&](int pass) {
        if (kind != MESH_BRICK)
            return pass ? shell_pass_ctas(md, pass) : kind == MESH_SHELL ? shell_stage_ctas(md) : arrays_stage_ctas(md);
        return hyper ? hyper_ctas(md, pass) : visc ? viscous_ctas(md, pass) : brick_stage_ctas(md);
    };
    const bool light = md->mesh->N == 2 && md->precision == CMDG_MIXED;
    auto before = [&](int pass) { return chain_releases(md->mesh->nelem, ctas(pass), light); };
    int flags = before(hyper || visc ? 1 : 0) ? RELEASE_STAGE : 0;
    if ((hyper || visc) && before(0)) flags |= RELEASE_PASS;
    if (hyper && before(2)) flags |= RELEASE_HYPER1;
    if (hyper && before(3)) flags |= RELEASE_HYPER2;
    md->release.store(flags, std::memory_order_relaxed);
    return flags;
}

KParams make_params(Model* md, const LaunchArgs& a) {
    const Mesh& m = *md->mesh;
    KParams P;
    P.Qin = a.Qin;
    P.Qout = a.Qout;
    P.dQ = a.dQ;
    P.emetric = m.d_emetric;
    P.nbr = m.d_nbr;
    P.lvl64 = md->d_lvl64;
    P.lvl32 = md->d_lvl32;
    P.jump32 = md->d_jump32;
    const bool mixed = md->precision == CMDG_MIXED;
    P.Dhat = mixed ? (const void*)md->d_Dhat32 : (const void*)md->d_Dhat64;
    P.status = md->d_status;
    P.nelem = (int)m.nelem;
    P.nz = m.nz;
    P.alpha = a.alpha;
    P.beta = a.beta;
    P.rka = a.rka;
    P.rkb_dt = a.rkb_dt;
    P.first_stage = a.first_stage;
    P.last_stage = a.last_stage;
    P.inv_w0 = 1.0 / m.omega[0];
    P.emetric32 = m.d_emetric32;
    P.rkb_dt32 = (float)a.rkb_dt;
    P.inv_w032 = (float)P.inv_w0;
    P.gm132 = (float)md->ph.gm1;
    P.gamma32 = (float)md->ph.gamma;
    P.ph = md->ph;
    for (int i = 0; i < (MAX_N + 1) * (MAX_N + 1); ++i) {
        const bool diag = i % (m.Nq + 1) == 0;
        P.DhatC64[i] = i < (int)m.Dhat.size() && !diag ? m.Dhat[i] : 0.0;
        P.DhatC32[i] = (float)P.DhatC64[i];
        P.DC64[i] = i < (int)m.D.size() && !diag ? m.D[i] : 0.0;
        P.DC32[i] = (float)P.DC64[i];
    }
    P.gf = md->d_gf;
    P.lvv64 = md->d_lvv64;
    P.lvv32 = md->d_lvv32;
    P.rho_nu32 = (float)md->ph.rho_nu;
    P.C_smag32 = (float)md->ph.C_smag;
    P.inv_Pr32 = (float)md->ph.inv_Pr_turb;
    P.kappa32 = (float)md->ph.kappa;
    P.MSLP32 = (float)md->ph.MSLP;
    P.grav32 = (float)md->ph.grav;
    P.geo = mixed ? (const void*)md->d_geo32 : (const void*)md->d_geo64;
    P.hd = md->d_hd;
    P.hlap = md->d_hlap;
    P.glap_ref32 = md->d_glap_ref;
    P.inv_tau_hyper = md->prm.tau_hyper > 0 ? 1.0 / md->prm.tau_hyper : 0.0;
    P.inv_tau_hyper32 = (float)P.inv_tau_hyper;
    P.nu4 = md->d_nu4;
    P.hyper_horizontal = md->prm.hyper_direction == CMDG_DIR_HORIZONTAL;
    P.fpart = m.d_fpart;
    P.fjump = md->d_fjump;
    P.hglap_ref32 = md->d_hglap_ref;
    P.vgref32 = md->d_vgref;
    P.sdelta = md->d_sdelta;
    P.mms_src = md->mms_src;
    P.mms_wall = md->mms_wall;
    P.mms_zero_h = md->mms_zero_h;
    P.cl_elem = md->d_cl_elem;
    P.wait_polls = md->wait_polls;
    P.staging_skip_copies = md->staging_skip_copies;
    P.backward = a.backward;
    P.release = chain_flags(md);
    return P;
}

int launch_stage(Model* md, const LaunchArgs& a, cudaStream_t s) {
    const Mesh& m = *md->mesh;
    if (m.kind == MESH_SHELL) return launch_shell_stage(md, a, s);
    if (m.kind == MESH_ARRAYS) {
        const cmdg_atmos_params& p = md->prm;
        if (!md->has_reference && (p.orientation != CMDG_ORIENT_NONE || p.gravity || p.ref_state)) {
            set_error("a model on a grid-arrays mesh needs cmdg_model_set_reference before its first tendency");
            return CMDG_ERR_STATE;
        }
        return launch_arrays_stage(md, a, s);
    }
    if (md->prm.hyperdiffusion != CMDG_HYPER_NONE) return launch_hyper_stage(md, a, s);
    if (md->prm.turbulence != CMDG_TURB_NONE) return launch_viscous_stage(md, a, s);
    const KParams P = make_params(md, a);
    const bool mixed = md->precision == CMDG_MIXED;
    cudaError_t err = cudaErrorNotSupported;
    if (md->kernel_kind == KERNEL_COLUMN) err = launch_column(P, m.N, mixed, a.mode, md->grid_ctas, s);
    if (md->kernel_kind == KERNEL_LINES) err = launch_lines(P, m.N, mixed, a.mode, s);
    if (md->kernel_kind == KERNEL_CLUSTER) {
        if (md->d_cl_elem == nullptr || md->cl_size != md->grid_ctas) {
            set_error("the cluster kernel needs its element map (cmdg_model_set_kernel)");
            return CMDG_ERR_STATE;
        }
        switch (m.N) {
            case 2: err = launch_cluster_N<2>(P, mixed, a.mode, md->cl_size, s); break;
            case 3: err = launch_cluster_N<3>(P, mixed, a.mode, md->cl_size, s); break;
            case 4: err = launch_cluster_N<4>(P, mixed, a.mode, md->cl_size, s); break;
            case 5: err = launch_cluster_N<5>(P, mixed, a.mode, md->cl_size, s); break;
            default: set_error("no kernel instantiated for N=%d", m.N); return CMDG_ERR_UNSUPPORTED;
        }
    }
    if (err == cudaErrorNotSupported) {
        switch (m.N) {
            case 2: err = launch_N<2>(P, mixed, a.mode, md->grid_ctas, s); break;
            case 3: err = launch_N<3>(P, mixed, a.mode, md->grid_ctas, s); break;
            case 4: err = launch_N<4>(P, mixed, a.mode, md->grid_ctas, s); break;
            case 5: err = launch_N<5>(P, mixed, a.mode, md->grid_ctas, s); break;
            default: set_error("no kernel instantiated for N=%d", m.N); return CMDG_ERR_UNSUPPORTED;
        }
    }
    if (err != cudaSuccess) {
        set_error("stage kernel launch failed: %s", cudaGetErrorString(err));
        return CMDG_ERR_CUDA;
    }
    return CMDG_OK;
}

cudaError_t launch_batch_stage(const KParams* d_params, const BatchTile* d_tiles, int ntiles, int N, int grid,
                               cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    switch (N) {
        case 3: return launch_batch_N<3>(d_params, d_tiles, ntiles, grid, s);
        case 4: return launch_batch_N<4>(d_params, d_tiles, ntiles, grid, s);
        case 5: return launch_batch_N<5>(d_params, d_tiles, ntiles, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_member_stage(const KParams& P, int N, cudaStream_t s) {
    switch (N) {
        case 3: return launch_N<3>(P, true, 1, -1, s);
        case 4: return launch_N<4>(P, true, 1, -1, s);
        case 5: return launch_N<5>(P, true, 1, -1, s);
        default: return cudaErrorInvalidValue;
    }
}

int batch_resident_ctas(int N) {
    switch (N) {
        case 3: return resident_N<3>();
        case 4: return resident_N<4>();
        case 5: return resident_N<5>();
        default: return 0;
    }
}

}  // namespace cmdg
