// tlw_volume.cuh -- fused per-element LW / MDRK volume kernels for TreeMesh{2} (FP64, sm_100a).
//
// Work split inside a CTA of EB whole elements (N=3: 8 x 16 nodes in 128 threads, N=4: 5 x 25 in 128,
// N=5: 3 x 36 in 128):
//  * node phase - one thread per GLL node ("owner") evaluates the Euler flux products at the perturbed states
//    (StencilSum) and keeps the LW stage state (u +- ut, u +- 2ut, the time averages F, G) in registers;
//  * line phase - each 1-D derivative contraction is done by one thread per (variable, element, line
//    index) that reads a whole row of f and a whole column of g from shared memory once, multiplies by
//    the derivative matrix held in constant memory (compile-time indices: the matrix entries are FMA
//    operands, no loads), and writes the row/column results back in place.
// Shared memory holds, per variable and element, a row-major plane of the node values with a padded
// plane stride chosen so that the owner accesses and the row/column accesses of the line phase are
// (nearly) bank-conflict free. Per stage a node writes 8 doubles and reads 8 back; a line reads and
// writes 2n. HBM traffic per element: read u once, write du (or u^{n+1}) once, write the face traces of
// U and F.n for the interface kernels.
//
// What bounds it (512^2, N = 4, one B200): the LSU data pipe (shared-memory wavefronts first), 65 % busy, beside the
// FP64 pipe (57 %) and the issue slots (55 %) at 20 warps an SM. Measured, this build against the one before the
// stencil sums: N = 3 0.251 -> 0.196 ms, N = 4 0.509 -> 0.431 ms, N = 5 0.809 -> 0.699 ms.
//
// Restates, per element (TreeMesh, no source terms):
//   LW depth 4 (N>=4): lw_volume_kernel_4!  src/solvers/dgsem_tree/dg_2d.jl:918-1249
//   LW depth 3 (N=3):  lw_volume_kernel_3!  src/solvers/dgsem_tree/dg_2d.jl:674-913
//   LW depth 2 (N=2):  lw_volume_kernel_2!  src/solvers/dgsem_tree/dg_2d.jl:495-669
//   LW depth 1 (N=1):  lw_volume_kernel_1!  src/solvers/dgsem_tree/dg_2d.jl:370-490
//   MDRK stage 1/2:    mdrk_kernel_1!/2!    src/solvers/dgsem_tree/multi_derivative_2d.jl:263-421, 423-555
// then the Trixi apply_jacobian! factor -J^{-1} is folded into the written result.
#pragma once
#include <type_traits>

#include "tlw_device.cuh"

namespace tlw {
// EBX = 0: the default number of elements per CTA; another value selects a tuned variant
// elements per CTA at N = 5: 3 (108 of 128 threads busy, 5 CTAs per SM): 0.740 ms the 512^2 kernel, against 0.752-0.763
// with 5, 7 or 8
#ifndef TLW_EB_N5
#define TLW_EB_N5 3
#endif
#ifndef TLW_VOLUME_MIN_BLOCKS
#define TLW_VOLUME_MIN_BLOCKS 5
#endif

template <int N, int EBX = 0>
struct VolCfg {
    static constexpr int n = N + 1;
    static constexpr int nn = n * n;
    // whole elements per CTA, chosen so that the CTA is (nearly) full warps
    static constexpr int EB = EBX ? EBX : N == 1 ? 32 : N == 2 ? 14 : N == 3 ? 8 : N == 4 ? 5 : N == 5 ? TLW_EB_N5 : N == 6 ? 5 : 2;
    static constexpr int THREADS = ((EB * nn + 31) / 32) * 32;
    // resident CTAs per SM the register allocation must allow (5 CTAs of 128 threads: <= 96 registers. 512^2, N = 4:
    // 0.465 ms, against 0.483 with 4 CTAs and 0.505 with 6, which spill; N = 3: 6 CTAs 0.232 against 0.213 ms)
    static constexpr int MIN_BLOCKS = THREADS <= 128 ? TLW_VOLUME_MIN_BLOCKS : 2;
    static constexpr int MDRK_MIN_BLOCKS = THREADS <= 128 ? 5 : 2;
    // curvilinear shock capturing (subcell normals, MUSCL face values): 4 CTAs of 128 threads, 128 registers
    static constexpr int SC_CURVED_MIN_BLOCKS = THREADS <= 128 ? 4 : 2;
    // plane layout: node (i, j) of (variable v, element e) at v*PV + e*P + i + R*j, on the Y planes of n = 4
    // transposed (YI, YJ); line threads take the variable innermost, then the element (LINE_E) or the line index.
    // P, PV and the order were chosen by counting the shared-memory wavefronts of the owner accesses and of the row
    // and column accesses (two a 64-bit warp access without conflicts). A contraction of a CTA then takes, against
    // element planes back to back with the line index innermost: N = 2 272 against 326, N = 3 256 (no conflicts)
    // against 320, N = 4 268 against 328, N = 5 292 against 340, N = 6 550 against 746, N = 7 320 against 768.
    static constexpr int R = n, YI = n == 4 ? n : 1, YJ = n == 4 ? 1 : n;
    static constexpr int P = n == 8 ? 65 : nn;
    static constexpr int PAD = n == 3 ? 6 : n == 4 ? 1 : n == 5 ? (EB % 2 ? 7 : 2) : n == 6 ? (EB > 3 ? 1 : 0) : n == 7 ? 7 : 0;
    static constexpr int PV = EB * P + PAD;
    static constexpr bool LINE_E = !(n == 4 || (n == 6 && EB == 3) || (n == 5 && EB == 10) || n == 7);
    // n = 4: a warp holds two whole elements, as nodes and as lines, so its phases need no CTA barrier
    static constexpr bool WARP_LOCAL = n == 4;
    static constexpr int PLANES = 4 * PV;              // doubles of one 4-variable field
    static constexpr int LINES = 4 * n * EB;           // (variable, element, line index)
    static constexpr int NODES = EB * nn;              // node slots of the CTA
    // doubles a node of the compact MDRK stage 2 keeps for itself (slot k of the node of thread t at k*NODES + t)
    static constexpr int MDRK_KEEP = 9;
    // regions: X (f / x-results), Y (g / y-results); shock capturing adds UU (u), VC (v1, v2, c, p),
    // FVX, FVY (first-order subcell fluxes), and with MUSCL subcells four regions of face values
    __host__ __device__ static constexpr size_t regions(bool sc, int rec) { return (size_t)(!sc ? 2 : rec ? 10 : 6) * PLANES; }
    static constexpr size_t lw_bytes(bool sc = false, int rec = 0) { return regions(sc, rec) * sizeof(double); }
    static constexpr size_t mdrk_bytes(bool sc = false, int rec = 0, bool compact = false) {
        return (regions(sc, rec) + (size_t)(compact ? MDRK_KEEP : 0) * NODES) * sizeof(double);
    }
};

// Taylor weights that are no short immediates: as constant operands they cost no instructions of their own (512^2,
// N = 4: 0.4366 -> 0.4325 ms)
static __constant__ double c_tlw_taylor[30] = {
    1.0, 1.0, 1.0 / 2.0, 1.0 / 6.0, 1.0 / 24.0,                  // 1 / M!
    2.0, 2.0, 4.0 / 3.0, 2.0 / 3.0,                              // 2^M / M!, M = 1..4
    0.25, 0.0, 0.0, 0.0,                                         // C_M / (M + 1)!, depth 1
    0.25, 1.0 / 6.0, 0.0, 0.0,                                   // depth 2
    1.0 / 24.0, 1.0 / 6.0, 1.0 / 48.0, 0.0,                      // depth 3
    1.0 / 24.0, 1.0 / 72.0, 1.0 / 48.0, 1.0 / 240.0,             // depth 4
    // int_0^1 of the quartic through its values at k = 0, 1, -1, 2, -2
    456.0 / 720.0, 346.0 / 720.0, -74.0 / 720.0, -19.0 / 720.0, 11.0 / 720.0};

enum VolMode { MODE_RHS = 0, MODE_STEP = 1 };

struct VolArgs {
    const double* u;        // state the stage fluxes are evaluated at  [v,i,j,e]
    const double* u_base;   // MODE_STEP, MDRK: out = u_base + dt * du  [v,i,j,e] (LW: u + dt * du)
    double* out;            // du (MODE_RHS) or the updated state (MODE_STEP)
    double* tU;             // face traces of U   [v, l, face, e]
    double* tF;             // face traces of F.n [v, l, face, e]
    double* tG;             // UnstructuredMesh2D: physical flux traces, tF <- F and tG <- G (null otherwise)
    // source terms (TreeMesh, FR volume integral): kind (1: source_terms_convergence_test), node coordinates
    // [2, i, j, e], the time of this rhs (device scalar), MDRK stage 1's S2 = s + s_t/6 [v, i, j, e]
    int source;
    const double* xnode;
    const double* tnow;
    double* S2;
    int compact;            // MDRK step on a plain TreeMesh: u_t between the stages instead of U2, F2
    double* U2;             // MDRK: stage-1 U2 [v,i,j,e] (written by stage 1, read by stage 2)
    double* F2;             // MDRK: stage-1 F2 [v,d,i,j,e]
    const double* inv_jac;  // [e]
    const double* dt;       // device scalar
    const Basis* basis;
    int E;
    double gamma, gm1, hg, inv_gamma;   // gamma, gamma - 1, (gamma - 1) / 2, 1 / gamma (set_gamma)
    void set_gamma(double g) { gamma = g; gm1 = g - 1.0; hg = 0.5 * gm1; inv_gamma = 1.0 / g; }
    // shock capturing (VolumeIntegralFRShockCapturing, first-order subcells)
    const double* alpha;    // blending factor per element
    double* tFn;            // first-order subcell flux next to each face [v, l, face, e] (fn_low)
    unsigned* status;
    int speed_kind;
    const int* inst;        // batched form: instance of each element (dt indexed by it); null otherwise
    // curvilinear meshes: contravariant vectors per node [4, i, j, e] (Ja^1_1, Ja^1_2, Ja^2_1, Ja^2_2) and the
    // inverse Jacobian per node [i, j, e] (inv_jac is then unused)
    const double* metrics;
    const double* inv_jac_node;
    unsigned long long* cfl_slots;   // plain step on a TreeMesh: per-element CFL slots (or null)
    int cfl_stride;                  // words per element there: CFL_SLOTS, or 2 (the interior maxima alone)
    unsigned* speed_status;          // status word of these speeds
    // BEGIN kernels (begin_step); null selects the others, whose dt is final
    StepState* step;
    unsigned long long* ring;
    unsigned long long* ring_next;
    // temporal error estimate of the Adaptive step control (lw_volume_kernel_4!'s u_np1 / u_np1_low tail)
    double* temporal_errors;          // [e]
    double abstol, reltol;
    double* dstore;                   // [m][e][v][node]: the stage derivatives d_1..d_depth (DSTORE kernels)
    // shock capturing on curvilinear meshes: subcell-face normals [e][d][line][f - 1][2] (d 0: xi faces on row
    // j, 1: eta faces on column i; f = 1..n-1), the normals the reference's calc_fn_low! takes for face n-1 of
    // pure DG elements [e][d][line][2], elements with a boundary face [e] (MUSCL: first order there), and the
    // MUSCL geometry: subcell faces [0..n] then the extended nodes [0..n+1] of the reference element
    const double* subn;
    const double* subq;
    const unsigned char* atb;
    const double* muscl_geom;
    int reconstruction;               // 0 first order, 1 MUSCL, 2 MUSCL-Hancock
};

// curvilinear: contravariant fluxes f~ = Ja^1_1 f + Ja^1_2 g, g~ = Ja^2_1 f + Ja^2_2 g of a node
// (contravariant_flux, src/solvers/dgsem_structured/dg_2d.jl:541-556)
__device__ __forceinline__ void contravariant(const double* Ja, const double* f, const double* g, double* ft,
                                              double* gt) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        ft[v] = fma(Ja[0], f[v], Ja[1] * g[v]);
        gt[v] = fma(Ja[2], f[v], Ja[3] * g[v]);
    }
}

// The records (K doubles a node) of the CTA that gets a free slot next, into L2: CTAs start in order, so that is the
// one as many further on as CTAs are resident, and its first loads then miss DRAM (512^2: N = 3 0.2143 -> 0.2105 ms,
// N = 4 0.4522 -> 0.4495, N = 5 0.7457 -> 0.7303). Threads ask for one 128-byte line each; nothing past the array.
template <class C>
__device__ __forceinline__ void prefetch_next(const double* p, int K, int E, int tid) {
    constexpr int AHEAD = 148 * C::MIN_BLOCKS;   // (SMs x CTAs)
    const size_t first = ((size_t)blockIdx.x + AHEAD) * C::NODES * K + (size_t)tid * 16;
    if (tid * 16 < C::NODES * K && first < (size_t)E * C::nn * K)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + first));
}

// BEGIN kernels, the first of a step that keeps its own CFL maximum: dt by one thread of each CTA before the CTA's first
// barrier, from the partial maxima at a.ring; block 0 leaves it in the step state and clears a.ring_next for this
// step's surface pass. Its loads and division hide behind the other warps' loads of u, and the step needs no dt launch
// (the rule that picks these kernels is begin_in_volume).
template <class C>
__device__ __forceinline__ void begin_step(const VolArgs& a, double* s_dt, int tid) {
    if (tid == 0) *s_dt = begin_step_dt(a.step, a.ring, a.ring_next, C::n, blockIdx.x == 0);
}
// barrier between the node phase and the line phase of the same elements
template <class C>
__device__ __forceinline__ void phase_sync() {
    if constexpr (C::WARP_LOCAL) __syncwarp();
    else __syncthreads();
}
// owner: the node's f and g into the contraction planes X and Y
template <int N, class C>
__device__ __forceinline__ void line_put(double* X, double* Y, int e, int i, int j, const double* f, const double* g) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        X[v * C::PV + e * C::P + i + C::R * j] = f[v];
        Y[v * C::PV + e * C::P + C::YI * i + C::YJ * j] = g[v];
    }
}
// owner: two fields of the node into two planes of the same layout
template <int N, class C>
__device__ __forceinline__ void node_put(double* X, double* Y, int e, int i, int j, const double* f, const double* g) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int a = v * C::PV + e * C::P + i + C::R * j;
        X[a] = f[v];
        Y[a] = g[v];
    }
}
// owner: x-result + y-result at the node
template <int N, class C>
__device__ __forceinline__ void node_sum(const double* X, const double* Y, int e, int i, int j, double* d) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int a = v * C::PV + e * C::P;
        d[v] = X[a + i + C::R * j] + Y[a + C::YI * i + C::YJ * j];
    }
}

// line phase, in place: X row (v,e,idx) <- M X row, Y column (v,e,idx) <- M Y column, with
// M = D (HAT = false) or Dhat (HAT = true):  x-result(i, j) = sum_k M[i,k] f(k, j),
// y-result(i, j) = sum_k M[j,k] g(i, k). Each row and column is read and written by one thread only.
// TLW_LINE_EVENODD = 1: lines of n >= 5 nodes take the even-odd form of M (c_tlw_D_eo / c_tlw_Dhat_eo), 2h^2 + 2h
// instead of n^2 multiply-adds per row (n = 5: 12 + 4 sums against 25); n <= 4 gains nothing and keeps M.
// Measured on the 512^2 steps (volume kernel, with the third-order reciprocal): N = 5 0.846 -> 0.809 ms, warped
// N = 4 0.535 -> 0.515 ms, N = 4 0.511 -> 0.509 ms; MDRK and shock capturing within 0.5 %.
#ifndef TLW_LINE_EVENODD
#define TLW_LINE_EVENODD 1
#endif
template <int N, class C, bool HAT>
__device__ __forceinline__ void line_contract_one(double* X, double* Y, int t) {
    constexpr int n = C::n;
    const int r = t >> 2;
    const int e = C::LINE_E ? r % C::EB : r / n, idx = C::LINE_E ? r / C::EB : r % n;
    const int pb = (t & 3) * C::PV + e * C::P;
    if constexpr (TLW_LINE_EVENODD && n >= 5) {
        constexpr int h = n / 2;
        constexpr int hh = h * h;
        const double* E = HAT ? c_tlw_Dhat_eo[N] : c_tlw_D_eo[N];
        // one line at a time (the row of X, then the column of Y) keeps the sums and differences of one line live,
        // not two
        auto line = [&](double* L, int base, int stride) {
            double a[n];
#pragma unroll
            for (int k = 0; k < n; ++k) a[k] = L[base + stride * k];
            double as[h], ad[h];
#pragma unroll
            for (int k = 0; k < h; ++k) {
                as[k] = a[k] + a[n - 1 - k];
                ad[k] = a[k] - a[n - 1 - k];
            }
#pragma unroll
            for (int o = 0; o < h; ++o) {
                double xa = E[o * h] * as[0], xb = E[hh + o * h] * ad[0];
#pragma unroll
                for (int k = 1; k < h; ++k) {
                    xa = fma(E[o * h + k], as[k], xa);
                    xb = fma(E[hh + o * h + k], ad[k], xb);
                }
                if constexpr (n % 2) xa = fma(E[2 * hh + o], a[h], xa);
                L[base + stride * o] = xb + xa;
                L[base + stride * (n - 1 - o)] = xb - xa;
            }
            if constexpr (n % 2) {
                double xm = E[2 * hh + h] * ad[0];
#pragma unroll
                for (int k = 1; k < h; ++k) xm = fma(E[2 * hh + h + k], ad[k], xm);
                L[base + stride * h] = xm;
            }
        };
        line(X, pb + C::R * idx, 1);
        line(Y, pb + idx, C::R);
    } else {
        const double* M = HAT ? c_tlw_Dhat[N] : c_tlw_D[N];
        double a[n], b[n];
#pragma unroll
        for (int k = 0; k < n; ++k) {
            a[k] = X[pb + k + C::R * idx];
            b[k] = Y[pb + C::YI * idx + C::YJ * k];
        }
#pragma unroll
        for (int o = 0; o < n; ++o) {
            double sx = 0.0, sy = 0.0;
#pragma unroll
            for (int k = 0; k < n; ++k) {
                sx = fma(M[o * n + k], a[k], sx);
                sy = fma(M[o * n + k], b[k], sy);
            }
            X[pb + o + C::R * idx] = sx;
            Y[pb + C::YI * idx + C::YJ * o] = sy;
        }
    }
}
template <int N, class C, bool HAT>
__device__ __forceinline__ void line_contract(double* X, double* Y, int tid) {
    if constexpr (C::LINES <= C::THREADS) {
        if (tid < C::LINES) line_contract_one<N, C, HAT>(X, Y, tid);
    } else {
#pragma unroll 1
        for (int t = tid; t < C::LINES; t += C::THREADS) line_contract_one<N, C, HAT>(X, Y, t);
    }
}

// ---- shock capturing helpers (src/solvers/dgsem_tree/dg_2d.jl:251-282, 1948-1991; Trixi calcflux_fv!) ----
// The subcell scheme works on the instantaneous u: each node parks u and (v1, v2, c, p), from which its right and upper
// neighbours form the fluxes of their common subcell faces (the shared-memory pipe bounds these kernels: the flux pairs
// at u parked as well, and both faces of a direction read back for the divergence, took 83 instead of 39 64-bit
// accesses a node; Riemann 256^2, N = 4: 152 -> 133 us). A node keeps the fluxes of its own left and lower face over
// the last contraction and reads the two others.
// stage 0: park u and (v1, v2, c, p)
template <int N, class C>
__device__ __forceinline__ void sc_park(double* UU, double* VC, int el, int i, int j, const double* u, double gamma,
                                        unsigned* status) {
    const double ir = nr_reciprocal(u[0]);
    const double v1 = u[1] * ir, v2 = u[2] * ir;
    const double p = (gamma - 1.0) * (u[3] - 0.5 * (u[1] * v1 + u[2] * v2));
    const double c = checked_sqrt(gamma * p * ir, status);
    const double vc[NV] = {v1, v2, c, p};
    node_put<N, C>(UU, VC, el, i, j, u, vc);
}
// what a subcell face needs of a node: the state, its velocity, sound speed and pressure
struct ScNode {
    double u[NV], v1, v2, c, p;
};
template <class C>
__device__ __forceinline__ ScNode sc_node(const double* UU, const double* VC, int at) {
    constexpr int PV = C::PV;
    return ScNode{{UU[at], UU[PV + at], UU[2 * PV + at], UU[3 * PV + at]}, VC[at], VC[PV + at], VC[2 * PV + at], VC[3 * PV + at]};
}
template <class C>
__device__ __forceinline__ ScNode sc_node(const double* u, const double* VC, int at, bool) {
    constexpr int PV = C::PV;
    return ScNode{{u[0], u[1], u[2], u[3]}, VC[at], VC[PV + at], VC[2 * PV + at], VC[3 * PV + at]};
}
// Rusanov (Trixi flux_lax_friedrichs, 4 arguments) across an x (D = 0) or y (D = 1) face
template <int D>
__device__ __forceinline__ void sc_face_flux(const ScNode& L, const ScNode& R, int speed_kind, double* out) {
    const double vL = D == 0 ? L.v1 : L.v2, vR = D == 0 ? R.v1 : R.v2;
    const double lambda = speed_kind == 0 ? fmax(fabs(vL), fabs(vR)) + fmax(L.c, R.c)
                                          : fmax(fabs(vL) + L.c, fabs(vR) + R.c);
    const double h = -0.5 * lambda;
    const double fL[NV] = {L.u[1 + D], fma(L.u[1], vL, D == 0 ? L.p : 0.0), fma(L.u[2], vL, D == 1 ? L.p : 0.0), (L.u[3] + L.p) * vL};
    const double fR[NV] = {R.u[1 + D], fma(R.u[1], vR, D == 0 ? R.p : 0.0), fma(R.u[2], vR, D == 1 ? R.p : 0.0), (R.u[3] + R.p) * vR};
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = 0.5 * (fL[v] + fR[v]) + h * (R.u[v] - L.u[v]);
}

// last contraction's input: each node computes the subcell flux on its left (fx) and lower (fy) subcell face. On
// elements that blend nothing in only those next to the element's faces, which the surface takes (fn_low [v, l, face, e]:
// faces -x, +x use the subcell faces between nodes 0|1 and n-2|n-1 of row j).
template <int N, class C>
__device__ __forceinline__ void sc_faces(const VolArgs& a, const double* UU, const double* VC, double* FVX, double* FVY,
                                         int el, int e, int i, int j, const double* u, bool blended, double* fx, double* fy) {
    constexpr int n = C::n, PV = C::PV;
    const int at = el * C::P + i + C::R * j;
    const bool edge_x = i == 1 || i == n - 1, edge_y = j == 1 || j == n - 1;
    const ScNode own = sc_node<C>(u, VC, at, true);
    const size_t tb = (size_t)e * 4 * n * NV;
    if (i >= 1 && (blended || edge_x)) {
        sc_face_flux<0>(sc_node<C>(UU, VC, at - 1), own, a.speed_kind, fx);
        if (edge_x) store4w(a.tFn + tb + ((i == 1 ? 0 : n) + j) * NV, fx);
        if (n == 2 && i == 1) store4w(a.tFn + tb + (n + j) * NV, fx);
#pragma unroll
        for (int v = 0; v < NV; ++v) FVX[v * PV + at] = fx[v];
    }
    if (j >= 1 && (blended || edge_y)) {
        sc_face_flux<1>(sc_node<C>(UU, VC, at - C::R), own, a.speed_kind, fy);
        if (edge_y) store4w(a.tFn + tb + ((j == 1 ? 2 * n : 3 * n) + i) * NV, fy);
        if (n == 2 && j == 1) store4w(a.tFn + tb + (3 * n + i) * NV, fy);
#pragma unroll
        for (int v = 0; v < NV; ++v) FVY[v * PV + at] = fy[v];
    }
}

// epilogue of a node with the weight alpha: fv = w_i^-1 (f*_{i+1/2} - f*_{i-1/2}) + w_j^-1 (g*_{j+1/2} - g*_{j-1/2})
// (element-boundary subcell fluxes are zero); acc <- (1 - alpha) acc + alpha fv
template <int N, class C>
__device__ __forceinline__ void sc_blend(const double* FVX, const double* FVY, int el, int i, int j, double alpha,
                                         const double* fx, const double* fy, double* acc) {
    constexpr int n = C::n, PV = C::PV;
    const int at = el * C::P + i + C::R * j;
    const double iwi = 1.0 / c_tlw_w[N][i], iwj = 1.0 / c_tlw_w[N][j];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const double xr = i + 1 < n ? FVX[v * PV + at + 1] : 0.0;
        const double yt = j + 1 < n ? FVY[v * PV + at + C::R] : 0.0;
        const double fv = iwi * (xr - (i >= 1 ? fx[v] : 0.0)) + iwj * (yt - (j >= 1 ? fy[v] : 0.0));
        acc[v] = (1.0 - alpha) * acc[v] + alpha * fv;
    }
}

// ---- shock capturing on curvilinear meshes, the reference's P4estMesh{2} path (src/solvers/dgsem_tree/
// dg_2d.jl:236-365, src/solvers/dgsem_structured/dg_2d.jl:75-311; Trixi calcflux_fv! for curved meshes) ----
// flux_lax_friedrichs(uL, uR, nrm)
__device__ __forceinline__ void sc_normal_flux(int speed_kind, const ScNode& L, const ScNode& R, const double* nrm, double* out) {
    const double nn = sqrt(nrm[0] * nrm[0] + nrm[1] * nrm[1]);
    const double vL = L.v1 * nrm[0] + L.v2 * nrm[1], vR = R.v1 * nrm[0] + R.v2 * nrm[1];
    const double lambda = speed_kind == 0 ? fmax(fabs(vL), fabs(vR)) + fmax(L.c, R.c) * nn
                                          : fmax(fabs(vL) + L.c * nn, fabs(vR) + R.c * nn);
    const double h = -0.5 * lambda;
    const double fL[NV] = {L.u[1] * nrm[0] + L.u[2] * nrm[1], fma(L.u[1], vL, L.p * nrm[0]), fma(L.u[2], vL, L.p * nrm[1]),
                           (L.u[3] + L.p) * vL};
    const double fR[NV] = {R.u[1] * nrm[0] + R.u[2] * nrm[1], fma(R.u[1], vR, R.p * nrm[0]), fma(R.u[2], vR, R.p * nrm[1]),
                           (R.u[3] + R.p) * vR};
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = 0.5 * (fL[v] + fR[v]) + h * (R.u[v] - L.u[v]);
}

// Julia sign
__device__ __forceinline__ double julia_sign(double x) { return (x == 0.0 || isnan(x)) ? x : (x > 0.0 ? 1.0 : -1.0); }

// minmod(a, b, 0) (src/solvers/dgsem_structured/dg_2d.jl:97-109): a NaN difference (0 / 0 at the element
// edges, where the extended state copies the edge node) has no sign equal to the other's and gives 0
__device__ __forceinline__ double minmod2(double a, double b) {
    const double slope = julia_min(fabs(a), fabs(b));
    const double s1 = julia_sign(a), s2 = julia_sign(b);
    if (s1 != s2) return 0.0;
    return s1 * slope;
}

// limit_variable_slope (src/equations/equations.jl:262-287), variable 0 density, 1 pressure
__device__ __forceinline__ double sc_limit_value(double gm1, int variable, const double* u) {
    return variable == 0 ? u[0] : gm1 * (u[3] - 0.5 * (u[1] * u[1] + u[2] * u[2]) / u[0]);
}
__device__ __forceinline__ void limit_variable_slope(double gm1, int variable, double* slope, double* usl, double* usr,
                                                     const double* ue, double xl, double xr) {
    const double vsl = sc_limit_value(gm1, variable, usl), vsr = sc_limit_value(gm1, variable, usr);
    const double vlow = sc_limit_value(gm1, variable, ue);
    const double threshold = 0.1 * vlow;
    if (vsl < 1e-10 || vsr < 1e-10) {
        const double rl = fabs(threshold - vlow) / (fabs(vsl - vlow) + 1e-13);
        const double rr = fabs(threshold - vlow) / (fabs(vsr - vlow) + 1e-13);
        const double theta = julia_min(julia_min(rl, rr), 1.0);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            slope[v] *= theta;
            usl[v] = ue[v] + (2.0 * theta) * (xl * slope[v]);
            usr[v] = ue[v] + (2.0 * theta) * (xr * slope[v]);
        }
    }
}

// Trixi flux(u, normal_direction, equations) of CompressibleEulerEquations2D
__device__ __forceinline__ void euler_flux_normal(double gm1, const double* u, const double* nrm, double* f) {
    const double rho = u[0], v1 = u[1] / rho, v2 = u[2] / rho;
    const double p = gm1 * (u[3] - 0.5 * (u[1] * v1 + u[2] * v2));
    const double vn = v1 * nrm[0] + v2 * nrm[1];
    const double rvn = rho * vn;
    f[0] = rvn;
    f[1] = rvn * v1 + p * nrm[0];
    f[2] = rvn * v2 + p * nrm[1];
    f[3] = (u[3] + p) * vn;
}

// minmod(a, b, c, beta, 0) (src/solvers/dgsem_structured/dg_2d.jl:83-95)
__device__ __forceinline__ double minmod3(double a, double b, double c, double beta) {
    const double slope = julia_min(julia_min(beta * fabs(a), fabs(b)), beta * fabs(c));
    const double s1 = julia_sign(a), s2 = julia_sign(b), s3 = julia_sign(c);
    if (s1 != s2 || s2 != s3) return 0.0;
    return s1 * slope;
}

// MUSCL (REC 1) and MUSCL-Hancock (REC 2) face values of node (i, j) into the UF regions k = 0 left, 1 right,
// 2 down, 3 up: slopes of the element-local extended state (calcflux_muscl! / calcflux_mh!,
// src/solvers/dgsem_structured/dg_2d.jl:196-253, 313-483: minmod of the one-sided differences, or with the centred
// one and beta = 2 - alpha for MUSCL-Hancock), limited for density then pressure (limit_slope,
// src/equations/compressible_euler_2d.jl:9-21). MUSCL-Hancock then adds to all four face values the multi-D
// half-step increments of the subcell, as the reference builds them: along xi +dt/2 J^{-1}(i, j) / w_{i+1}
// f(left).n_i (1 <= i <= n-2) and -dt/2 J^{-1}(i, j) / w_{i+1} f(right).n_{i+1} (i <= n-2); along eta the
// same with J^{-1}(i, j+1) (dt_fv: the time step fv_kernel! is given).
template <int N, class C, int REC>
__device__ __forceinline__ void sc_muscl_faces(const VolArgs& a, const double* UU, double* UF, int el, int e, int i,
                                               int j, double gm1, double alpha, double dt_fv, double ij) {
    constexpr int n = C::n, nn = n * n;
    constexpr int PV = C::PV;
    const double* sf = a.muscl_geom;           // subcell faces [0..n]
    const double* xe = a.muscl_geom + n + 1;   // extended nodes [0..n+1]
    auto at = [&](int ii, int jj, int v) {
        ii = ii < 0 ? 0 : (ii > n - 1 ? n - 1 : ii);
        jj = jj < 0 ? 0 : (jj > n - 1 ? n - 1 : jj);
        return UU[v * PV + el * C::P + ii + C::R * jj];
    };
    const int I = i + 1, J = j + 1;
    const double h1x = __ldg(xe + I) - __ldg(xe + I - 1), h2x = __ldg(xe + I + 1) - __ldg(xe + I);
    const double h1y = __ldg(xe + J) - __ldg(xe + J - 1), h2y = __ldg(xe + J + 1) - __ldg(xe + J);
    double u_[NV], sx[NV], sy[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        u_[v] = at(i, j, v);
        const double ul = at(i - 1, j, v), ur = at(i + 1, j, v), ud = at(i, j - 1, v), uu = at(i, j + 1, v);
        if (REC == 1) {
            sx[v] = minmod2((u_[v] - ul) / h1x, (ur - u_[v]) / h2x);
            sy[v] = minmod2((u_[v] - ud) / h1y, (uu - u_[v]) / h2y);
        } else {
            // finite_differences (dg_2d.jl:75-81)
            const double beta = 2.0 - alpha;
            const double ax = -(h2x / (h1x * (h1x + h2x))), bx = (h2x - h1x) / (h1x * h2x), cx = (h1x / (h2x * (h1x + h2x)));
            const double ay = -(h2y / (h1y * (h1y + h2y))), by = (h2y - h1y) / (h1y * h2y), cy = (h1y / (h2y * (h1y + h2y)));
            sx[v] = minmod3((u_[v] - ul) / h1x, ax * ul + bx * u_[v] + cx * ur, (ur - u_[v]) / h2x, beta);
            sy[v] = minmod3((u_[v] - ud) / h1y, ay * ud + by * u_[v] + cy * uu, (uu - u_[v]) / h2y, beta);
        }
    }
    const double xl = __ldg(sf + I - 1) - __ldg(xe + I), xr = __ldg(sf + I) - __ldg(xe + I);
    const double yl = __ldg(sf + J - 1) - __ldg(xe + J), yr = __ldg(sf + J) - __ldg(xe + J);
    double fv[4][NV];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        double* s = d == 0 ? sx : sy;
        const double lo = d == 0 ? xl : yl, hi = d == 0 ? xr : yr;
        double pa[NV], pb[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            pa[v] = u_[v] + 2.0 * s[v] * lo;
            pb[v] = u_[v] + 2.0 * s[v] * hi;
        }
        limit_variable_slope(gm1, 0, s, pa, pb, u_, lo, hi);
        limit_variable_slope(gm1, 1, s, pa, pb, u_, lo, hi);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            fv[2 * d][v] = u_[v] + s[v] * lo;
            fv[2 * d + 1][v] = u_[v] + s[v] * hi;
        }
    }
    if (REC == 2) {
        // increments in the reference's order: xi "rr", xi "ll", eta "uu", eta "dd"
        double inc[4][NV];
        const double ijn = j + 1 < n ? __ldg(a.inv_jac_node + (size_t)e * nn + i + n * (j + 1)) : 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int d = q >> 1, c = d == 0 ? i : j, line = d == 0 ? j : i;
            // q 0: the cell's own face c (its left / lower value, +), q 1: face c + 1 (right / upper value, -)
            const int f = (q & 1) ? c + 1 : c;
            const bool on = (q & 1) ? c <= n - 2 : (c >= 1 && c <= n - 2);
            double r[NV] = {0.0, 0.0, 0.0, 0.0};
            if (on) {
                const double* np = a.subn + ((((size_t)e * 2 + d) * n + line) * (n - 1) + (f - 1)) * 2;
                const double nrm[2] = {__ldg(np), __ldg(np + 1)};
                double fl[NV];
                euler_flux_normal(gm1, fv[2 * d + (q & 1)], nrm, fl);
                const double jj = d == 0 ? ij : ijn;
                const double cf = ((q & 1) ? -0.5 : 0.5) * dt_fv * jj / c_tlw_w[N][c + 1];
#pragma unroll
                for (int v = 0; v < NV; ++v) r[v] = cf * fl[v];
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) inc[q][v] = r[v];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int v = 0; v < NV; ++v) fv[k][v] = (((fv[k][v] + inc[0][v]) + inc[1][v]) + inc[2][v]) + inc[3][v];
    }
    const int o = el * C::P + i + C::R * j;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int v = 0; v < NV; ++v) UF[k * C::PLANES + v * PV + o] = fv[k][v];
}

// last contraction's input on a curvilinear mesh: the subcell flux on the node's left (xi) and lower (eta) face along
// the subcell normal; pure DG elements only need faces 1 and n-1, the latter with the reference's calc_fn_low! normal;
// MUSCL elements take the reconstructed face values. fn_low of the four faces in load_fn_low!'s P4estMesh order (slot 0
// bottom, 1 right, 2 top, 3 left).
template <int N, class C, int REC>
__device__ __forceinline__ void sc_faces_curved(const VolArgs& a, const double* UU, const double* VC, const double* UF,
                                                double* FVX, double* FVY, int el, int e, int i, int j, const double* u,
                                                bool blended, bool muscl, double* fx, double* fy) {
    constexpr int n = C::n;
    constexpr int PV = C::PV;
    const size_t tb = (size_t)e * 4 * n * NV;
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const int f = d == 0 ? i : j, line = d == 0 ? j : i;
        if (f < 1 || (!blended && f != 1 && f != n - 1)) continue;
        const double* np = (!blended && f == n - 1)
                               ? a.subq + (((size_t)e * 2 + d) * n + line) * 2
                               : a.subn + ((((size_t)e * 2 + d) * n + line) * (n - 1) + (f - 1)) * 2;
        const double nrm[2] = {__ldg(np), __ldg(np + 1)};
        const int aR = el * C::P + i + C::R * j, aL = aR - (d == 0 ? 1 : C::R);
        ScNode L, R;
        if (REC >= 1 && muscl) {
            // the right (up) face value of the node before the face, the left (down) one of the node after it
            const double* PL = UF + (d == 0 ? 1 : 3) * C::PLANES;
            const double* PR = UF + (d == 0 ? 0 : 2) * C::PLANES;
#pragma unroll
            for (int v = 0; v < NV; ++v) { L.u[v] = PL[v * PV + aL]; R.u[v] = PR[v * PV + aR]; }
            for (ScNode* q : {&L, &R}) {
                const double ir = 1.0 / q->u[0];
                q->v1 = q->u[1] * ir;
                q->v2 = q->u[2] * ir;
                q->p = a.gm1 * (q->u[3] - 0.5 * (q->u[1] * q->v1 + q->u[2] * q->v2));
                q->c = checked_sqrt(a.gamma * q->p * ir, a.status);
            }
        } else {
            L = sc_node<C>(UU, VC, aL);
            R = sc_node<C>(u, VC, aR, true);
        }
        double* out = d == 0 ? fx : fy;
        sc_normal_flux(a.speed_kind, L, R, nrm, out);
        if (f == 1 || f == n - 1) store4w(a.tFn + tb + ((d == 0 ? (i == 1 ? 3 : 1) : (j == 1 ? 0 : 2)) * n + line) * NV, out);
        double* dst = d == 0 ? FVX : FVY;
#pragma unroll
        for (int v = 0; v < NV; ++v) dst[v * PV + aR] = out[v];
    }
}

// epilogue on a curvilinear mesh: acc <- (1 - alpha) acc (+ alpha fv on blended elements)
template <int N, class C>
__device__ __forceinline__ void sc_blend_curved(const double* FVX, const double* FVY, int el, int i, int j, double alpha,
                                                bool blended, const double* fx, const double* fy, double* acc) {
    if (blended) {
        sc_blend<N, C>(FVX, FVY, el, i, j, alpha, fx, fy, acc);
    } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = (1.0 - alpha) * acc[v];
    }
}

// The face traces [v, l, face, e] of U and F.n of a node (faces -x, +x, -y, +y), written as soon as U, F, G are formed,
// so that they are not held over the last contraction. One store for the two x faces and one for the two y faces: a
// 256-bit warp store costs eight wavefronts however few lanes are active.
template <int n>
__device__ __forceinline__ void store_traces(const VolArgs& a, int e, int i, int j, const double* U, const double* F,
                                             const double* G) {
    const size_t tb = (size_t)e * 4 * n * NV;
    const bool nf = a.tG == nullptr;   // UnstructuredMesh2D: the flux traces were written before (physical)
    if (i == 0 || i == n - 1) {
        const size_t k = tb + ((i == 0 ? 0 : n) + j) * NV;
        store4w(a.tU + k, U);
        if (nf) store4w(a.tF + k, F);
    }
    if (j == 0 || j == n - 1) {
        const size_t k = tb + ((j == 0 ? 2 * n : 3 * n) + i) * NV;
        store4w(a.tU + k, U);
        if (nf) store4w(a.tF + k, G);
    }
}

// The node's result: o = s acc (+ S), the rhs (MODE_RHS, s = -J^{-1}), or base + s acc (+ dt S), the updated state
// (MODE_STEP, s = -dt J^{-1}). acc = Dhat-contraction of (F, G), S the source's time average.
template <int MODE>
__device__ __forceinline__ void store_result(double* out, double s, double dt, const double* acc, const double* base,
                                             const double* S, double* o) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (MODE == MODE_RHS) o[v] = S ? s * acc[v] + S[v] : s * acc[v];   // (S enters unscaled by J^{-1})
        else o[v] = fma(s, acc[v], S ? fma(dt, S[v], base[v]) : base[v]);
    }
    store4w(out, o);
}

// UnstructuredMesh2D: the physical time-averaged fluxes F (x) and G (y) on every face the node lies on, which its
// interfaces dot with the caller's normals (prolong2interfaces!, src/solvers/dgsem_unstructured_2d/dg_2d.jl:60-200)
template <int n>
__device__ __forceinline__ void physical_flux_traces(const VolArgs& a, int e, int i, int j, const double* F,
                                                     const double* G) {
    const size_t tb = (size_t)e * 4 * n * NV;
    if (i == 0) { store4(a.tF + tb + (0 * n + j) * NV, F); store4(a.tG + tb + (0 * n + j) * NV, G); }
    if (i == n - 1) { store4(a.tF + tb + (1 * n + j) * NV, F); store4(a.tG + tb + (1 * n + j) * NV, G); }
    if (j == 0) { store4(a.tF + tb + (2 * n + i) * NV, F); store4(a.tG + tb + (2 * n + i) * NV, G); }
    if (j == n - 1) { store4(a.tF + tb + (3 * n + i) * NV, F); store4(a.tG + tb + (3 * n + i) * NV, G); }
}

// ---- source terms (calc_source / calc_source_t_N12 ... _tttt_N4, src/solvers/dgsem_tree/dg_2d.jl:89-175) ----
// Kind 1, Trixi's source_terms_convergence_test for CompressibleEulerEquations2D: the source of the manufactured
// solution rho = rho v1 = rho v2 = c + A sin(w (x + y - t)), rho e = rho^2 (c = 2, A = 0.1, w = 2 pi / L, L = 2):
// with rho' = w A cos(w (x + y - t)) and tmp = (2 rho - 1)(gamma - 1), s = (rho', rho' (1 + tmp), rho' (1 + tmp),
// 2 rho' (rho + tmp)). It does not depend on u, so every stencil of the reference is a combination of
// s(x, t + k dt), k = -2..2, and the reference's argument-order slips in two of its calls (dg_2d.jl:891-897,
// :1227-1233: states in the wrong slots) leave the values unchanged.
struct SrcNode {
    double x1, x2, t, dt, gamma;
};
__device__ __forceinline__ void src_eval(const SrcNode& q, double k, double* s) {
    const double w = 2.0 * 3.14159265358979323846 * (1.0 / 2.0);
    const double arg = w * (q.x1 + q.x2 - (q.t + k * q.dt));
    const double si = sin(arg), co = cos(arg);
    const double rho = 2.0 + 0.1 * si;
    const double rho_x = w * 0.1 * co;
    const double tmp = (2.0 * rho - 1.0) * (q.gamma - 1.0);
    s[0] = rho_x;
    s[1] = rho_x * (1.0 + tmp);
    s[2] = s[1];
    s[3] = 2.0 * rho_x * (rho + tmp);
}
// o = c * sum_k w_k s(t + k dt), k = -2..2 (zero weights skipped)
__device__ __forceinline__ void src_term(const SrcNode& q, double w, double k, double* acc) {
    if (w == 0.0) return;
    double s[NV];
    src_eval(q, k, s);
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = fma(w, s[v], acc[v]);
}
__device__ __forceinline__ void src_stencil(const SrcNode& q, double c, double wm2, double wm1, double w0, double wp1,
                                            double wp2, double* o) {
    double acc[NV] = {0.0, 0.0, 0.0, 0.0};
    src_term(q, wm2, -2.0, acc);
    src_term(q, wm1, -1.0, acc);
    src_term(q, w0, 0.0, acc);
    src_term(q, wp1, 1.0, acc);
    src_term(q, wp2, 2.0, acc);
#pragma unroll
    for (int v = 0; v < NV; ++v) o[v] = c * acc[v];
}
// the reference's stencils (each with its own time offsets)
__device__ __forceinline__ void src_t_N12(const SrcNode& q, double* o) { src_stencil(q, 0.5, 0.0, -1.0, 0.0, 1.0, 0.0, o); }
__device__ __forceinline__ void src_t_N34(const SrcNode& q, double* o) {
    src_stencil(q, 1.0 / 12.0, 1.0, -8.0, 0.0, 8.0, -1.0, o);
}
__device__ __forceinline__ void src_tt_N23(const SrcNode& q, double* o) { src_stencil(q, 1.0, 0.0, 1.0, -2.0, 1.0, 0.0, o); }
__device__ __forceinline__ void src_tt_N4(const SrcNode& q, double* o) {
    src_stencil(q, 1.0 / 12.0, -1.0, 16.0, -30.0, 16.0, -1.0, o);
}
__device__ __forceinline__ void src_ttt_N34(const SrcNode& q, double* o) {
    src_stencil(q, 0.5, -1.0, 2.0, 0.0, -2.0, 1.0, o);
}
__device__ __forceinline__ void src_tttt_N4(const SrcNode& q, double* o) {
    src_stencil(q, 1.0, 1.0, -4.0, 6.0, -4.0, 1.0, o);
}

// The per-element CFL slots of a step's final values (plain TreeMesh step): after the epilogue, every thread has
// the speeds of its node in l1, l2 (interior nodes; zero otherwise); through the (now free) X plane, one thread per
// (element, component) writes slot 0 (interior maxima) and clears the face slots, which the surfaces fill.
// Every thread of the CTA calls it (barriers inside).
template <int N, class C>
__device__ __forceinline__ void write_interior_slots(const VolArgs& a, double* X, bool active, int el, int i, int j,
                                                     int tid, double l1, double l2) {
    constexpr int n = C::n, EB = C::EB;
    __syncthreads();
    if (active) {
        X[el * C::P + i + C::R * j] = l1;
        X[(EB + el) * C::P + i + C::R * j] = l2;
    }
    __syncthreads();
    const int ee = blockIdx.x * EB + (tid >> 1);
    if (tid < 2 * EB && ee < a.E) {
        const double* p = X + ((tid & 1) * EB + (tid >> 1)) * C::P;
        double m = 0.0;
#pragma unroll
        for (int jj = 1; jj < n - 1; ++jj)
#pragma unroll
            for (int ii = 1; ii < n - 1; ++ii) m = fmax(m, p[ii + C::R * jj]);
        unsigned long long* sl = a.cfl_slots + (size_t)ee * a.cfl_stride;
        sl[tid & 1] = (unsigned long long)__double_as_longlong(m);
        if (a.cfl_stride == CFL_SLOTS) {
#pragma unroll
            for (int k = 1; k < CFL_SLOTS / 2; ++k) sl[2 * k + (tid & 1)] = 0ull;
        }
    }
}

// Flux pairs and their stencils. The stencils of the time derivatives of f and g are sums over the perturbed states
// of products, of which five differ: rho v1^2, rho v2^2, rho v1 v2, H v1 and H v2 (H = rho e + p); what is linear in
// the state (rho v1, rho v2 and the rho e part of p) has a stencil of L times the current derivative d of the state,
// L the stencil's moment, so it is not summed at all: f = (L d_2, a + P, b, x), g = (L d_3, b, c + P, y) with
// P = (gamma - 1)(L d_4 - (a + c) / 2). A state carries gamma rho e as its last variable, so that H is one multiply-add.
// A stage of four pairs then takes 64 FP64 instructions instead of 96 (N = 4: about 730 -> 626 a node, counted). Summing
// rho |v|^2 in the place of rho v2^2 saves 4 of them and no time (512^2 5071 against 5078 us a pass of 8 steps, warped
// 201 x 167 880 against 872), but rounds the small flux of rho v2 by the large one of a stream along x: at Mach 30 the
// error of its rhs is 2 to 2.5 times that of the mirrored stream (N = 3, 4, 5).
struct StencilSum {
    double a, c, b, x, y;
};
// the products at p plus (SGN = 1) or minus (SGN = -1) those at m; hg = (gamma - 1) / 2, irp, irm = 1 / rho
template <int SGN>
__device__ __forceinline__ StencilSum stencil_pair(double hg, const double* p, double irp, const double* m, double irm) {
    const double v1 = p[1] * irp, v2 = p[2] * irp, w1 = m[1] * irm, w2 = m[2] * irm;
    const double ap = p[1] * v1, am = m[1] * w1, cp = p[2] * v2, cm = m[2] * w2;
    const double hp = fma(-hg, ap + cp, p[3]), hm = SGN * fma(-hg, am + cm, m[3]);
    return StencilSum{fma((double)SGN, am, ap), fma((double)SGN, cm, cp), fma(SGN * m[1], w2, p[1] * v2),
                      fma(hm, w1, hp * v1), fma(hm, w2, hp * v2)};
}
__device__ __forceinline__ StencilSum stencil_fma(double c, const StencilSum& t, const StencilSum& q) {   // c t + q
    return StencilSum{fma(c, t.a, q.a), fma(c, t.c, q.c), fma(c, t.b, q.b), fma(c, t.x, q.x), fma(c, t.y, q.y)};
}
__device__ __forceinline__ StencilSum stencil_fmsub(double c, const StencilSum& t, const StencilSum& q) {  // c t - q
    return StencilSum{fma(c, t.a, -q.a), fma(c, t.c, -q.c), fma(c, t.b, -q.b), fma(c, t.x, -q.x), fma(c, t.y, -q.y)};
}
__device__ __forceinline__ void stencil_fluxes(double gm1, double hg, double L, const StencilSum& r, const double* d,
                                               double* f, double* g) {
    const double P = fma(-hg, r.a + r.c, gm1 * (L * d[3]));
    f[0] = L * d[1]; f[1] = r.a + P; f[2] = r.b; f[3] = r.x;
    g[0] = L * d[2]; g[1] = r.b; g[2] = r.c + P; g[3] = r.y;
}
// the flux pair at u (unscaled rho e) and its products
__device__ __forceinline__ StencilSum flux_base(double gm1, const double* u, double* f, double* g) {
    const double ir = nr_reciprocal(u[0]);
    const double v1 = u[1] * ir, v2 = u[2] * ir;
    const double a = u[1] * v1, c = u[2] * v2, b = u[1] * v2;
    const double p = gm1 * fma(-0.5, a + c, u[3]), h = u[3] + p;
    f[0] = u[1]; f[1] = a + p; f[2] = b; f[3] = h * v1;
    g[0] = u[2]; g[1] = b; g[2] = c + p; g[3] = h * v2;
    return StencilSum{a, c, b, f[3], g[3]};
}

// the four reciprocals of a stage first, as independent chains
struct Recip4 {
    double pp, p, m, mm;
};
__device__ __forceinline__ Recip4 recip4(const double* upp, const double* up, const double* um, const double* umm) {
    Recip4 r;
    r.pp = nr_reciprocal(upp[0]);
    r.p = nr_reciprocal(up[0]);
    r.m = nr_reciprocal(um[0]);
    r.mm = nr_reciprocal(umm[0]);
    return r;
}
// the stencil of f_t, g_t at u +- d, u +- 2d times 12 (-f(u+2d) + 8 f(u+d) - 8 f(u-d) + f(u-2d)): an MDRK stage
__device__ __forceinline__ void first_derivative_fluxes(const VolArgs& a, const double* u, const double* d, double* f,
                                                        double* g) {
    const double us[NV] = {u[0], u[1], u[2], a.gamma * u[3]}, ds[NV] = {d[0], d[1], d[2], a.gamma * d[3]};
    double up[NV], um[NV], upp[NV], umm[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        up[v] = us[v] + ds[v];
        um[v] = us[v] - ds[v];
        upp[v] = fma(2.0, ds[v], us[v]);
        umm[v] = fma(-2.0, ds[v], us[v]);
    }
    const Recip4 rc = recip4(upp, up, um, umm);
    const StencilSum t = stencil_pair<-1>(a.hg, up, rc.p, um, rc.m);
    const StencilSum q = stencil_pair<-1>(a.hg, upp, rc.pp, umm, rc.mm);
    stencil_fluxes(a.gm1, a.hg, 12.0, stencil_fmsub(8.0, t, q), d, f, g);
}

// ------------------------------------------------------------------------------------------------
// Plain LW volume kernel (depth = min(N, 4)).
// The finite-difference stencils are accumulated unscaled ("raw"); their constant factors and -dt J^{-1}
// are applied to the contraction result (s below) and folded into the F/G update coefficients:
//   depth 4: f_t = raw1/12, f_tt = raw2/12, f_ttt = raw3/2, f_tttt = raw4/2
//   depth 3: f_t = raw1/12, f_tt = raw2,    f_ttt = raw3/2
//   depth 2: f_t = raw1/2,  f_tt = raw2;    depth 1: f_t = raw1/2
// ------------------------------------------------------------------------------------------------
// DSTORE: also write each stage derivative d_m (dt-scaled time derivative of u) to a.dstore, for the discrete
// adjoint's reverse sweep, which then reads them instead of recomputing them. Layout [m][e][v][node]: one
// element's d_m is contiguous (a bulk copy per tile of elements) with the nodes innermost (conflict-free
// shared-memory reads, one thread per node).
template <int nn>
__device__ __forceinline__ void store_stage_derivative(const VolArgs& a, int m, long long e, int node, const double* d) {
    double* p = a.dstore + ((size_t)(m - 1) * a.E + e) * NV * nn + node;
#pragma unroll
    for (int v = 0; v < NV; ++v) p[v * nn] = d[v];
}

// REC (curvilinear shock capturing): 0 first-order subcells, 1 MUSCL subcells
// SRC: source terms (a.source, FR volume integral): S = s + s_t/2 + s_tt/6 + ... with each stencil added to its time
// derivative (dt s_k) before the perturbed states move, and S enters the update unscaled by J^{-1}. The curvilinear
// kernel of depth 4 takes the 5-point s_tt (calc_source_tt_N4, dgsem_structured/dg_2d.jl:1886) where the TreeMesh
// one takes the 3-point calc_source_tt_N23 (dgsem_tree/dg_2d.jl:1093-1104).
template <int N, int MODE, bool SC, int EBX = 0, bool CURVED = false, bool TE = false, bool DSTORE = false, int REC = 0,
          bool SRC = false, bool BEGIN = false>
static __global__ void __launch_bounds__(VolCfg<N, EBX>::THREADS, (SC && CURVED) ? VolCfg<N, EBX>::SC_CURVED_MIN_BLOCKS
                                                                  : SRC ? VolCfg<N, EBX>::MDRK_MIN_BLOCKS - 1
                                                                        : VolCfg<N, EBX>::MIN_BLOCKS)
    lw_volume_kernel(VolArgs a) {
    static_assert(REC == 0 || (SC && CURVED), "MUSCL subcells: curvilinear shock capturing");
    static_assert(!SRC || (!SC && !TE && !DSTORE), "source terms: the FR volume integral, without the error estimate");
    static_assert(!BEGIN || (MODE == MODE_STEP && !SC && !CURVED && !TE && !DSTORE && !SRC), "dt in the kernel: the plain step");
    // the temporal error estimate of the Adaptive step control: the TreeMesh computes it at depth 4 only
    // (lw_volume_kernel_3! of dgsem_tree has none), the curvilinear kernels at depths 3 and 4
    static_assert(!TE || (CURVED ? N >= 3 : N >= 4), "temporal errors: TreeMesh N >= 4, curvilinear N >= 3");
    static_assert(!DSTORE || (!SC && !CURVED && !TE), "stored stage derivatives: the plain TreeMesh kernel");
    using C = VolCfg<N, EBX>;
    constexpr int n = C::n, nn = C::nn, EB = C::EB;
    constexpr int DEPTH = N >= 4 ? 4 : N;
    constexpr double C1 = DEPTH >= 3 ? 1.0 / 12.0 : 0.5;
    constexpr double C2 = DEPTH == 4 ? 1.0 / 12.0 : 1.0;
    constexpr double C3 = 0.5;
    constexpr double C4 = 0.5;
    extern __shared__ double smem_d[];
    double* X = smem_d;
    double* Y = X + C::PLANES;
    double* UU = Y + C::PLANES;        // shock capturing only: u, (v1, v2, c, p), subcell fluxes
    double* VC = UU + C::PLANES;
    double* FVX = VC + C::PLANES;
    double* FVY = FVX + C::PLANES;
    double* UF = FVY + C::PLANES;      // curvilinear MUSCL: face values, 4 regions (left, right, down, up)

    const int tid = threadIdx.x;
    wait_for_previous();
    if (!SC) dependents_may_start();
    prefetch_next<C>(a.u, 4, a.E, tid);
    if (CURVED) {
        prefetch_next<C>(a.metrics, 4, a.E, tid);
        prefetch_next<C>(a.inv_jac_node, 1, a.E, tid);
    }
    const int el = tid / nn;
    const int node = tid - el * nn;
    const int i = node % n, j = node / n;
    const int e = blockIdx.x * EB + el;
    const bool active = el < EB && e < a.E;
    // shock capturing: DG only where alpha is 0 (curvilinear: within 1e-12 of it, pure_and_blended_element_ids!); MUSCL
    // subcells on blended elements without a boundary face
    double alpha_e = 0.0, fx[NV], fy[NV];
    bool blended = false, muscl = false;
    if (SC && active) {
        alpha_e = a.alpha[e];
        blended = CURVED ? !(fabs(alpha_e) <= 1e-12) : alpha_e != 0.0;
        muscl = CURVED && REC >= 1 && blended && !__ldg(a.atb + e);
    }
    double dt = 0.0;
    __shared__ double s_dt;
    if constexpr (BEGIN) begin_step<C>(a, &s_dt, tid);
    else dt = a.inst ? a.dt[__ldg(a.inst + min(e, a.E - 1))] : *a.dt;
    // per-element maxima of the interior nodes' speeds for the next step's CFL (plain LW step only)
    constexpr bool SLOTS = MODE == MODE_STEP && !SC && !TE;

    // F[1..3] and G[2], G[3] are accumulated stage by stage; F[0], G[0] (the time averages of rho v1, rho v2) follow
    // from U, and G[1] = F[2]. The states carry gamma rho e as their last variable (see StencilSum).
    double U[NV], F[NV], G[NV], up[NV], um[NV], upp[NV], umm[NV];
    double Ssrc[NV] = {0.0, 0.0, 0.0, 0.0};   // SRC: the source's time average S
    SrcNode sq{};
    double s0 = 0.0;             // -dt J^{-1} (of the element, or of the node on curvilinear meshes)
    double dF[NV], dG[NV];       // TE: the last stage's term of F, G
    double ub[NV];               // u again, from the last stage on (the states' registers are free then)
    auto inverse_jacobian = [&]() {
        return CURVED ? __ldg(a.inv_jac_node + (size_t)e * nn + node) : __ldg(a.inv_jac + e);
    };
    // stage fluxes into the contraction planes (contravariant on curvilinear meshes, whose metric terms come from L1
    // each time: held in registers they spilled, warped 201 x 167, N = 4)
    auto put = [&](const double* f, const double* g) {
        if (CURVED) {
            double ft[NV], gt[NV], Ja[4];
            load4w_const(a.metrics + ((size_t)e * nn + node) * 4, Ja);
            contravariant(Ja, f, g, ft, gt);
            line_put<N, C>(X, Y, el, i, j, ft, gt);
        } else {
            line_put<N, C>(X, Y, el, i, j, f, g);
        }
    };
    // u again where it is needed (from L1): the pass is bound by the shared-memory pipe, on which a global record
    // costs as much as four 64-bit loads, and the products of the flux pair at u are cheaper formed again than kept
    auto load_u = [&](double* uu) { load4w(a.u + ((size_t)e * nn + node) * NV, uu); };
    // stage 0: f, g at u (dg_2d.jl:941-971; dgsem_structured/dg_2d.jl:1709-1740)
    if (active) {
        double uu[NV], f[NV], g[NV];
        load4w(a.u + ((size_t)e * nn + node) * NV, uu);
        s0 = BEGIN ? -inverse_jacobian() : -dt * inverse_jacobian();   // (BEGIN: dt after the first barrier)
        if (SRC) {
            // S = s(u, x, t) (dg_2d.jl:979-987)
            const double* xn = a.xnode + 2 * ((size_t)e * nn + node);
            sq = SrcNode{__ldg(xn), __ldg(xn + 1), *a.tnow, dt, a.gamma};
            src_eval(sq, 0.0, Ssrc);
        }
        flux_base(a.gm1, uu, f, g);
        put(f, g);
        if (SC) sc_park<N, C>(UU, VC, el, i, j, uu, a.gamma, a.status);
        uu[3] *= a.gamma;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            F[v] = f[v]; G[v] = g[v];
            up[v] = um[v] = upp[v] = umm[v] = uu[v];
        }
    }

    // stage M (dg_2d.jl:972-1206; depth 3 :725-875, depth 2 :543-634, depth 1 :417-454): the M-th derivative d of u
    // (times dt^M), the perturbed states u + k d_1 + ... + k^M / M! d_M, k = +-1, +-2, and the stencil of their fluxes
    auto stage = [&](auto stage_number) {
        constexpr int M = decltype(stage_number)::value;
        constexpr double CM[5] = {1.0, C1, C2, C3, C4};
        constexpr double LM[5] = {0.0, DEPTH >= 3 ? 12.0 : 2.0, DEPTH == 4 ? 12.0 : 1.0, 2.0, 1.0};
        constexpr double SIGN = M % 2 ? -1.0 : 1.0;
        const double W1 = c_tlw_taylor[M], W2 = c_tlw_taylor[4 + M];
        if (BEGIN && M == 1) {
            __syncthreads();
            dt = s_dt;
            s0 *= dt;
        } else {
            phase_sync<C>();
        }
        line_contract<N, C, false>(X, Y, tid);
        phase_sync<C>();
        if (M == 1 && SC && CURVED && REC >= 1 && muscl) sc_muscl_faces<N, C, REC>(a, UU, UF, el, e, i, j, a.gm1, alpha_e, dt, inverse_jacobian());
        if (!active) return;
        if (M == 2 || M == DEPTH) load_u(ub);
        double d[NV], f[NV], g[NV];
        node_sum<N, C>(X, Y, el, i, j, d);
        const double s = s0 * CM[M - 1];
        double sk[NV];
        if (SRC && M == 2) {   // s_t from the states after ut: N34 at depths 3, 4, N12 at depth 2 (dg_2d.jl:1027-1040)
            if (DEPTH >= 3) src_t_N34(sq, sk);
            else src_t_N12(sq, sk);
        } else if (SRC && M == 3) {   // s_tt: N23 on the TreeMesh (dg_2d.jl:1093-1104), N4 on curvilinear depth 4
            if (CURVED && DEPTH == 4) src_tt_N4(sq, sk);
            else src_tt_N23(sq, sk);
        } else if (SRC && M == 4) {
            src_ttt_N34(sq, sk);      // s_ttt (dg_2d.jl:1148-1162)
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            d[v] *= s;
            if (SRC && M > 1) Ssrc[v] = fma(W1, sk[v], Ssrc[v]);
            if (SRC) d[v] = fma(dt, M == 1 ? Ssrc[v] : sk[v], d[v]);
        }
        if (DSTORE) store_stage_derivative<nn>(a, M, e, node, d);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double dv = v == 3 ? a.gamma * d[3] : d[v];
            up[v] = fma(W1, dv, up[v]);
            um[v] = fma(SIGN * W1, dv, um[v]);
            if (DEPTH >= 3) {
                upp[v] = fma(W2, dv, upp[v]);
                umm[v] = fma(SIGN * W2, dv, umm[v]);
            }
        }
        StencilSum r, f0;
        if (M == 2 || M == 4) f0 = flux_base(a.gm1, ub, f, g);
        if (DEPTH >= 3) {
            const Recip4 rc = recip4(upp, up, um, umm);
            const StencilSum t = stencil_pair<M % 2 ? -1 : 1>(a.hg, up, rc.p, um, rc.m);
            if (M == 2 && DEPTH == 3) {
                r = stencil_fma(-2.0, f0, t);                     // f(up) - 2 f0 + f(um)
            } else {
                const StencilSum q = stencil_pair<M % 2 ? -1 : 1>(a.hg, upp, rc.pp, umm, rc.mm);
                if (M == 1) r = stencil_fmsub(8.0, t, q);                // -f(upp) + 8 f(up) - 8 f(um) + f(umm)
                else if (M == 2) r = stencil_fma(16.0, t, stencil_fmsub(-30.0, f0, q));
                                                                         // -f(upp) + 16 f(up) - 30 f0 + 16 f(um) - f(umm)
                else if (M == 3) r = stencil_fma(-2.0, t, q);            // f(upp) - 2 f(up) + 2 f(um) - f(umm)
                else r = stencil_fma(-4.0, t, stencil_fma(6.0, f0, q));
                                                                         // f(upp) - 4 f(up) + 6 f0 - 4 f(um) + f(umm)
            }
        } else {
            const double rp = nr_reciprocal(up[0]), rm = nr_reciprocal(um[0]);
            r = stencil_pair<M % 2 ? -1 : 1>(a.hg, up, rp, um, rm);        // f(up) - f(um)
            if (M == 2) r = stencil_fma(-2.0, f0, r);             // f(up) - 2 f0 + f(um)
        }
        stencil_fluxes(a.gm1, a.hg, LM[M], r, d, f, g);
        const double WC = c_tlw_taylor[9 + (DEPTH - 1) * 4 + M - 1];
#pragma unroll
        for (int v = 1; v < NV; ++v) F[v] = fma(WC, f[v], F[v]);
#pragma unroll
        for (int v = 2; v < NV; ++v) G[v] = fma(WC, g[v], G[v]);
        if (TE && M == DEPTH) {
#pragma unroll
            for (int v = 0; v < NV; ++v) { dF[v] = WC * f[v]; dG[v] = WC * g[v]; }
        }
        if (M < DEPTH) {
            put(f, g);
        } else {
            // U = int_0^1 of the polynomial through the states at k = -2..2 (or -1..1)
            const double uu[NV] = {ub[0], ub[1], ub[2], a.gamma * ub[3]};
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                if (DEPTH >= 3)
                    U[v] = fma(c_tlw_taylor[25], uu[v], fma(c_tlw_taylor[26], up[v], fma(c_tlw_taylor[27], um[v],
                           fma(c_tlw_taylor[28], upp[v], c_tlw_taylor[29] * umm[v]))));
                else
                    U[v] = fma(8.0 / 12.0, uu[v], fma(5.0 / 12.0, up[v], (-1.0 / 12.0) * um[v]));
            }
            U[3] *= a.inv_gamma;
            // the flux of rho is rho v1 (rho v2): its time average is U's, up to the stencil's factor C4 of f_tttt
            constexpr double WU = DEPTH == 4 ? (C4 - 1.0) / 120.0 : 0.0;
            F[0] = fma(WU, d[1], U[1]);
            G[0] = fma(WU, d[2], U[2]);
            G[1] = F[2];
        }
    };
    stage(std::integral_constant<int, 1>{});
    if constexpr (DEPTH >= 2) stage(std::integral_constant<int, 2>{});
    if constexpr (DEPTH >= 3) stage(std::integral_constant<int, 3>{});
    if constexpr (DEPTH >= 4) stage(std::integral_constant<int, 4>{});
    // final: Dhat contraction of the time-averaged fluxes (every owner has read its node's results of
    // the last contraction before writing F, G over them: same address, same thread)
    if (SRC && active) {
        // the last stencil: depth 1 s_t / 2 (N12), 2 s_tt / 6 (N23), 3 s_ttt / 24, 4 s_tttt / 120
        // (dg_2d.jl:474-477, :651-654, :891-897, :1227-1233)
        double sk[NV];
        if (DEPTH == 1) src_t_N12(sq, sk);
        else if (DEPTH == 2) src_tt_N23(sq, sk);
        else if (DEPTH == 3) src_ttt_N34(sq, sk);
        else src_tttt_N4(sq, sk);
        const double c = DEPTH == 1 ? 0.5 : DEPTH == 2 ? 1.0 / 6.0 : DEPTH == 3 ? 1.0 / 24.0 : 1.0 / 120.0;
#pragma unroll
        for (int v = 0; v < NV; ++v) Ssrc[v] = fma(c, sk[v], Ssrc[v]);
    }
    if (active) {
        if (CURVED) {
            if (a.tG) physical_flux_traces<n>(a, e, i, j, F, G);
            // the surface needs the normal fluxes: keep the contravariant time averages F~, G~ (their face
            // values are F . Ja^1 and F . Ja^2)
            double ft[NV], gt[NV], Ja[4];
            load4w_const(a.metrics + ((size_t)e * nn + node) * 4, Ja);
            contravariant(Ja, F, G, ft, gt);
#pragma unroll
            for (int v = 0; v < NV; ++v) { F[v] = ft[v]; G[v] = gt[v]; }
            if (TE) {   // the last stage's term of F~, G~
                contravariant(Ja, dF, dG, ft, gt);
#pragma unroll
                for (int v = 0; v < NV; ++v) { dF[v] = ft[v]; dG[v] = gt[v]; }
            }
        }
        store_traces<n>(a, e, i, j, U, F, G);
        line_put<N, C>(X, Y, el, i, j, F, G);
        if (SC) {
            if constexpr (CURVED) sc_faces_curved<N, C, REC>(a, UU, VC, UF, FVX, FVY, el, e, i, j, ub, blended, muscl, fx, fy);
            else sc_faces<N, C>(a, UU, VC, FVX, FVY, el, e, i, j, ub, blended, fx, fy);
        }
    }
    phase_sync<C>();
    line_contract<N, C, true>(X, Y, tid);
    phase_sync<C>();
    double l1 = 0.0, l2 = 0.0;
    if (active) {
        double acc[NV], o[NV];
        node_sum<N, C>(X, Y, el, i, j, acc);
        if (SC) {
            if constexpr (CURVED) sc_blend_curved<N, C>(FVX, FVY, el, i, j, alpha_e, blended, fx, fy, acc);
            else if (blended) sc_blend<N, C>(FVX, FVY, el, i, j, alpha_e, fx, fy, acc);
        }
        store_result<MODE>(a.out + ((size_t)e * nn + node) * NV, MODE == MODE_STEP ? s0 : -inverse_jacobian(), dt, acc, ub,
                           SRC ? Ssrc : nullptr, o);
        if (SLOTS && a.cfl_slots && i > 0 && i < n - 1 && j > 0 && j < n - 1) {
            node_speeds(a.gamma, o, a.speed_status, l1, l2);
            if (CURVED) {
                const size_t k = (size_t)e * nn + node;
                double Jn[4];
                load4w_const(a.metrics + k * 4, Jn);
                curved_speeds(Jn, __ldg(a.inv_jac_node + k), l1, l2);
            }
        }
    }
    if (SLOTS && a.cfl_slots) write_interior_slots<N, C>(a, X, active, el, i, j, tid, l1, l2);
    if (TE) {
        // lw_volume_kernel_4!'s error estimate (dg_2d.jl:1183-1265; curvilinear, with F~, G~ and the node's
        // J^{-1}: dgsem_structured/dg_2d.jl:1595-1682 at depth 3, :1983-2075 at depth 4): the strong-form volume
        // updates u_np1 = u - dt J^{-1} (D F + D G) and u_np1_low with F, G before the last stage's term;
        // temporal_errors[e] = sum over nodes and variables of ((u_np1 - u_np1_low) / (abstol + reltol max))^2
        double un[NV], err = 0.0;
        phase_sync<C>();
        if (active) line_put<N, C>(X, Y, el, i, j, F, G);
        phase_sync<C>();
        line_contract<N, C, false>(X, Y, tid);
        phase_sync<C>();
        if (active) {
            double dd[NV];
            node_sum<N, C>(X, Y, el, i, j, dd);
#pragma unroll
            for (int v = 0; v < NV; ++v) un[v] = fma(s0, dd[v], ub[v]);
        }
        phase_sync<C>();
        if (active) line_put<N, C>(X, Y, el, i, j, dF, dG);
        phase_sync<C>();
        line_contract<N, C, false>(X, Y, tid);
        phase_sync<C>();
        if (active) {
            double dd[NV];
            node_sum<N, C>(X, Y, el, i, j, dd);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const double lo = un[v] - s0 * dd[v];
                const double r = (un[v] - lo) / (a.abstol + a.reltol * fmax(fabs(un[v]), fabs(lo)));
                err = fma(r, r, err);
            }
        }
        phase_sync<C>();
        if (active) X[el * C::P + i + C::R * j] = err;
        __syncthreads();
        const int ee = blockIdx.x * EB + tid;
        if (tid < EB && ee < a.E) {
            double sum = 0.0;
            for (int jj = 0; jj < n; ++jj)
                for (int ii = 0; ii < n; ++ii) sum += X[tid * C::P + ii + C::R * jj];
            a.temporal_errors[ee] = sum;
        }
    }
}

// MDRK stage 1's stored sums from u^n and d = u_t: F2 = f + f_t/6, G2 = g + g_t/6, U2 = u + u_t/6 with f_t the
// 4-point stencil at u +- d, u +- 2d (multi_derivative_2d.jl:337-371), the operations of mdrk1_volume_kernel
__device__ __forceinline__ void mdrk_stage1_sums(const VolArgs& a, const double* uu, const double* d, double* F2v,
                                                 double* G2v, double* U2v) {
    double f0[NV], g0[NV], ft[NV], gt[NV];
    flux_base(a.gm1, uu, f0, g0);
    first_derivative_fluxes(a, uu, d, ft, gt);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        F2v[v] = fma(1.0 / 72.0, ft[v], f0[v]);
        G2v[v] = fma(1.0 / 72.0, gt[v], g0[v]);
        U2v[v] = fma(1.0 / 6.0, d[v], uu[v]);
    }
}

// ------------------------------------------------------------------------------------------------
// MDRK stage 1 (mdrk_kernel_1!, multi_derivative_2d.jl:263-421): F = f/2 + f_t/8, U = u/2 + u_t/8,
// F2 = f + f_t/6, U2 = u + u_t/6 (stored whole for stage 2).
// ------------------------------------------------------------------------------------------------
// CURVED (mdrk_kernel_1!, src/solvers/dgsem_structured/multi_derivative_2d.jl:82-243): the contractions take the
// contravariant fluxes, d carries the node's J^{-1}; F2, G2 stay physical, the traces are contravariant.
// SRC (FR volume integral): ut += dt s(u, t); S = s/2 + s_t/8 enters du, S2 = s + s_t/6 is stored for stage 2
// (multi_derivative_2d.jl:321-400; dgsem_structured/multi_derivative_2d.jl:151-239).
// COMPACT (the plain TreeMesh step): store only u_t (into a.U2) instead of U2 and F2; stage 2 recomputes them from
// u^n and u_t with this kernel's operations (64 instead of 192 bytes a node between the stages).
template <int N, int MODE, bool SC, bool CURVED = false, int REC = 0, bool SRC = false, bool COMPACT = false,
          bool BEGIN = false>
static __global__ void __launch_bounds__(VolCfg<N>::THREADS, (SC && CURVED) ? VolCfg<N>::SC_CURVED_MIN_BLOCKS
                                                                         : VolCfg<N>::MDRK_MIN_BLOCKS)
    mdrk1_volume_kernel(VolArgs a) {
    static_assert(!BEGIN || COMPACT, "dt in the kernel: the plain step");
    static_assert(REC == 0 || (SC && CURVED), "MUSCL subcells: curvilinear shock capturing");
    static_assert(!SRC || !SC, "source terms: the FR volume integral");
    static_assert(!COMPACT || (!SC && !CURVED && !SRC && MODE == MODE_STEP), "compact stages: the plain TreeMesh step");
    using C = VolCfg<N>;
    constexpr int n = C::n, nn = C::nn, EB = C::EB;
    extern __shared__ double smem_d[];
    double* X = smem_d;
    double* Y = X + C::PLANES;
    double* UU = Y + C::PLANES;        // shock capturing only: u, (v1, v2, c, p), subcell fluxes
    double* VC = UU + C::PLANES;
    double* FVX = VC + C::PLANES;
    double* FVY = FVX + C::PLANES;
    double* UF = FVY + C::PLANES;      // curvilinear MUSCL: face values, 4 regions (left, right, down, up)
    const int tid = threadIdx.x;
    wait_for_previous();
    if (!SC) dependents_may_start();
    prefetch_next<C>(a.u, 4, a.E, tid);
    const int el = tid / nn;
    const int node = tid - el * nn;
    const int i = node % n, j = node / n;
    const int e = blockIdx.x * EB + el;
    const bool active = el < EB && e < a.E;
    double alpha_e = 0.0, fx[NV], fy[NV];
    bool blended = false, muscl = false;
    if (SC && active) {
        alpha_e = a.alpha[e];
        blended = CURVED ? !(fabs(alpha_e) <= 1e-12) : alpha_e != 0.0;
        muscl = CURVED && REC >= 1 && blended && !__ldg(a.atb + e);
    }
    double dt = 0.0;
    __shared__ double s_dt;
    if constexpr (BEGIN) begin_step<C>(a, &s_dt, tid);
    else dt = a.inst ? a.dt[__ldg(a.inst + min(e, a.E - 1))] : *a.dt;
    double uu[NV], f0[NV], g0[NV], ij = 0.0, Ja[4] = {0.0, 0.0, 0.0, 0.0};
    // a flux pair into the contraction planes (contravariant on curvilinear meshes)
    auto put = [&](const double* f, const double* g) {
        if (CURVED) {
            double ft[NV], gt[NV];
            contravariant(Ja, f, g, ft, gt);
            line_put<N, C>(X, Y, el, i, j, ft, gt);
        } else {
            line_put<N, C>(X, Y, el, i, j, f, g);
        }
    };
    if (active) {
        load4w(a.u + ((size_t)e * nn + node) * NV, uu);
        if (CURVED) {
            load4w_const(a.metrics + ((size_t)e * nn + node) * 4, Ja);
            ij = __ldg(a.inv_jac_node + (size_t)e * nn + node);
        } else {
            ij = __ldg(a.inv_jac + e);
        }
        flux_base(a.gm1, uu, f0, g0);
        put(f0, g0);
        if (SC) {
            // the subcell FV part uses the instantaneous u^n (multi_derivative_2d.jl:205)
            sc_park<N, C>(UU, VC, el, i, j, uu, a.gamma, a.status);
        }
    }
    if (BEGIN) {
        __syncthreads();
        dt = s_dt;
    } else {
        phase_sync<C>();
    }
    // (the MUSCL face values are read by the neighbours after the next barrier)
    if (SC && CURVED && REC >= 1 && muscl) sc_muscl_faces<N, C, REC>(a, UU, UF, el, e, i, j, a.gm1, alpha_e, 0.5 * dt, ij);
    line_contract<N, C, false>(X, Y, tid);
    phase_sync<C>();
    double U[NV], F[NV], G[NV], Ssrc[NV] = {0.0, 0.0, 0.0, 0.0};
    if (active) {
        double d[NV], ft[NV], gt[NV];
        node_sum<N, C>(X, Y, el, i, j, d);
        const double s0 = -dt * ij;
#pragma unroll
        for (int v = 0; v < NV; ++v) d[v] *= s0;
        SrcNode sq{};
        double sn[NV];
        if (SRC) {
            const double* xn = a.xnode + 2 * ((size_t)e * nn + node);
            sq = SrcNode{__ldg(xn), __ldg(xn + 1), *a.tnow, dt, a.gamma};
            src_eval(sq, 0.0, sn);
#pragma unroll
            for (int v = 0; v < NV; ++v) d[v] = fma(dt, sn[v], d[v]);
        }
        first_derivative_fluxes(a, uu, d, ft, gt);
        double U2v[NV], F2v[NV], G2v[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            F[v] = fma(0.125 / 12.0, ft[v], 0.5 * f0[v]);
            G[v] = fma(0.125 / 12.0, gt[v], 0.5 * g0[v]);
            U[v] = fma(0.125, d[v], 0.5 * uu[v]);
            F2v[v] = fma(1.0 / 72.0, ft[v], f0[v]);
            G2v[v] = fma(1.0 / 72.0, gt[v], g0[v]);
            U2v[v] = fma(1.0 / 6.0, d[v], uu[v]);
        }
        const size_t off = ((size_t)e * nn + node);
        if (COMPACT) {
            store4w(a.U2 + off * NV, d);
        } else {
            store4w(a.U2 + off * NV, U2v);
            store4w(a.F2 + off * 2 * NV, F2v);
            store4w(a.F2 + off * 2 * NV + NV, G2v);
        }
        if (SRC) {
            double st[NV], S2v[NV];
            src_t_N34(sq, st);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                Ssrc[v] = fma(0.125, st[v], 0.5 * sn[v]);
                S2v[v] = fma(1.0 / 6.0, st[v], sn[v]);
            }
            store4w(a.S2 + off * NV, S2v);
        }
        if (CURVED) {
            double ft2[NV], gt2[NV];
            contravariant(Ja, F, G, ft2, gt2);
#pragma unroll
            for (int v = 0; v < NV; ++v) { F[v] = ft2[v]; G[v] = gt2[v]; }
        }
        store_traces<n>(a, e, i, j, U, F, G);
        line_put<N, C>(X, Y, el, i, j, F, G);
        if (SC) {
            if constexpr (CURVED) sc_faces_curved<N, C, REC>(a, UU, VC, UF, FVX, FVY, el, e, i, j, uu, blended, muscl, fx, fy);
            else sc_faces<N, C>(a, UU, VC, FVX, FVY, el, e, i, j, uu, blended, fx, fy);
        }
    }
    phase_sync<C>();
    line_contract<N, C, true>(X, Y, tid);
    phase_sync<C>();
    if (active) {
        double acc[NV];
        node_sum<N, C>(X, Y, el, i, j, acc);
        if (SC) {
            if constexpr (CURVED) sc_blend_curved<N, C>(FVX, FVY, el, i, j, alpha_e, blended, fx, fy, acc);
            else if (blended) sc_blend<N, C>(FVX, FVY, el, i, j, alpha_e, fx, fy, acc);
        }
        double o[NV], ub[NV];
        if (MODE == MODE_STEP) load4w(a.u_base + ((size_t)e * nn + node) * NV, ub);
        store_result<MODE>(a.out + ((size_t)e * nn + node) * NV, MODE == MODE_STEP ? -dt * ij : -ij, dt, acc, ub,
                           SRC ? Ssrc : nullptr, o);
    }
}

// ------------------------------------------------------------------------------------------------
// MDRK stage 2 (mdrk_kernel_2!, multi_derivative_2d.jl:423-555): at u* = a.u,
// F = F2 + f_t(u*)/3, U = U2 + u*_t/3.
// ------------------------------------------------------------------------------------------------
// CURVED (mdrk_kernel_2!, src/solvers/dgsem_structured/multi_derivative_2d.jl:245-445): as in stage 1.
// SRC (FR volume integral): u*_t += dt s(u*); S = S2 + s_t(u*)/3 (multi_derivative_2d.jl:484-550), the source at
// t + dt/2 on the TreeMesh and at t on curvilinear meshes (dgsem_structured/multi_derivative_2d.jl:325-361).
// COMPACT: F2, G2, U2 recomputed from u^n (a.u_base) and stage 1's u_t (a.U2) at the start, parked in the node's
// shared-memory slots until the stage's own sums are formed.
template <int N, int MODE, bool SC, bool CURVED = false, int REC = 0, bool SRC = false, bool COMPACT = false>
static __global__ void __launch_bounds__(VolCfg<N>::THREADS, (SC && CURVED) ? VolCfg<N>::SC_CURVED_MIN_BLOCKS
                                                                         : VolCfg<N>::MDRK_MIN_BLOCKS)
    mdrk2_volume_kernel(VolArgs a) {
    static_assert(REC == 0 || (SC && CURVED), "MUSCL subcells: curvilinear shock capturing");
    static_assert(!SRC || !SC, "source terms: the FR volume integral");
    static_assert(!COMPACT || (!SC && !CURVED && !SRC && MODE == MODE_STEP), "compact stages: the plain TreeMesh step");
    using C = VolCfg<N>;
    constexpr int n = C::n, nn = C::nn, EB = C::EB;
    extern __shared__ double smem_d[];
    double* X = smem_d;
    double* Y = X + C::PLANES;
    double* UU = Y + C::PLANES;        // shock capturing only: u, (v1, v2, c, p), subcell fluxes
    double* VC = UU + C::PLANES;
    double* FVX = VC + C::PLANES;
    double* FVY = FVX + C::PLANES;
    double* UF = FVY + C::PLANES;      // curvilinear MUSCL: face values, 4 regions (left, right, down, up)
    const int tid = threadIdx.x;
    wait_for_previous();
    if (!SC) dependents_may_start();
    prefetch_next<C>(a.u, 4, a.E, tid);
    if (COMPACT) {
        prefetch_next<C>(a.u_base, 4, a.E, tid);
        prefetch_next<C>(a.U2, 4, a.E, tid);
    }
    const int el = tid / nn;
    const int node = tid - el * nn;
    const int i = node % n, j = node / n;
    const int e = blockIdx.x * EB + el;
    const bool active = el < EB && e < a.E;
    double alpha_e = 0.0, fx[NV], fy[NV];
    bool blended = false, muscl = false;
    if (SC && active) {
        alpha_e = a.alpha[e];
        blended = CURVED ? !(fabs(alpha_e) <= 1e-12) : alpha_e != 0.0;
        muscl = CURVED && REC >= 1 && blended && !__ldg(a.atb + e);
    }
    // dt of this element's instance (batched form) or the single dt
    const double dt = a.inst ? a.dt[__ldg(a.inst + min(e, a.E - 1))] : *a.dt;
    double* keep = smem_d + C::regions(SC, REC) + tid;   // COMPACT: the node's slots
    constexpr int K = C::NODES;
    double us[NV], ij = 0.0, Ja[4] = {0.0, 0.0, 0.0, 0.0};
    if (active) {
        double f[NV], g[NV];
        load4w(a.u + ((size_t)e * nn + node) * NV, us);
        if (CURVED) {
            load4w_const(a.metrics + ((size_t)e * nn + node) * 4, Ja);
            ij = __ldg(a.inv_jac_node + (size_t)e * nn + node);
        } else {
            ij = __ldg(a.inv_jac + e);
        }
        euler_fluxes(a.gm1, us[0], us[1], us[2], us[3], f, g);
        if (CURVED) {
            double ft[NV], gt[NV];
            contravariant(Ja, f, g, ft, gt);
            line_put<N, C>(X, Y, el, i, j, ft, gt);
        } else {
            line_put<N, C>(X, Y, el, i, j, f, g);
        }
        if (COMPACT) {
            // stage 1's U2, F2 and G2 from u^n and u_t (F2 and G2 of rho are U2 of rho v1, rho v2), in the node's slots
            double un[NV], dn[NV], F2v[NV], G2v[NV], U2v[NV];
            const size_t off = ((size_t)e * nn + node);
            load4w(a.u_base + off * NV, un);
            load4w(a.U2 + off * NV, dn);
            mdrk_stage1_sums(a, un, dn, F2v, G2v, U2v);
#pragma unroll
            for (int v = 0; v < NV; ++v) keep[v * K] = U2v[v];
            keep[4 * K] = F2v[1]; keep[5 * K] = F2v[2]; keep[6 * K] = F2v[3];
            keep[7 * K] = G2v[2]; keep[8 * K] = G2v[3];
        }
        if (SC) {
            // the subcell FV part uses the instantaneous u^n, not u* (multi_derivative_2d.jl:257)
            double un[NV];
            load4w(a.u_base + ((size_t)e * nn + node) * NV, un);
            sc_park<N, C>(UU, VC, el, i, j, un, a.gamma, a.status);
        }
    }
    phase_sync<C>();
    // (the MUSCL face values are read by the neighbours after the next barrier)
    if (SC && CURVED && REC >= 1 && muscl) sc_muscl_faces<N, C, REC>(a, UU, UF, el, e, i, j, a.gm1, alpha_e, dt, ij);
    line_contract<N, C, false>(X, Y, tid);
    phase_sync<C>();
    double U[NV], F[NV], G[NV], Ssrc[NV] = {0.0, 0.0, 0.0, 0.0};
    if (active) {
        double d[NV], ft[NV], gt[NV];
        node_sum<N, C>(X, Y, el, i, j, d);
        const double s0 = -dt * ij;
#pragma unroll
        for (int v = 0; v < NV; ++v) d[v] *= s0;
        if (SRC) {
            const double* xn = a.xnode + 2 * ((size_t)e * nn + node);
            // at t + dt/2 on the TreeMesh (multi_derivative_2d.jl:484-495), at t on curvilinear meshes
            // (dgsem_structured/multi_derivative_2d.jl:336, 361)
            const SrcNode sq{__ldg(xn), __ldg(xn + 1), CURVED ? *a.tnow : *a.tnow + 0.5 * dt, dt, a.gamma};
            double sn[NV], st[NV];
            src_eval(sq, 0.0, sn);
#pragma unroll
            for (int v = 0; v < NV; ++v) d[v] = fma(dt, sn[v], d[v]);
            src_t_N34(sq, st);
            load4w(a.S2 + ((size_t)e * nn + node) * NV, sn);
#pragma unroll
            for (int v = 0; v < NV; ++v) Ssrc[v] = fma(1.0 / 3.0, st[v], sn[v]);
        }
        first_derivative_fluxes(a, us, d, ft, gt);
        const size_t off = ((size_t)e * nn + node);
        double U2v[NV], F2v[NV], G2v[NV];
        if (COMPACT) {
#pragma unroll
            for (int v = 0; v < NV; ++v) U2v[v] = keep[v * K];
            F2v[0] = U2v[1]; F2v[1] = keep[4 * K]; F2v[2] = keep[5 * K]; F2v[3] = keep[6 * K];
            G2v[0] = U2v[2]; G2v[1] = F2v[2]; G2v[2] = keep[7 * K]; G2v[3] = keep[8 * K];
        } else {
            load4w(a.U2 + off * NV, U2v);
            load4w(a.F2 + off * 2 * NV, F2v);
            load4w(a.F2 + off * 2 * NV + NV, G2v);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            F[v] = fma(1.0 / 36.0, ft[v], F2v[v]);
            G[v] = fma(1.0 / 36.0, gt[v], G2v[v]);
            U[v] = fma(1.0 / 3.0, d[v], U2v[v]);
        }
        if (CURVED) {
            double ft2[NV], gt2[NV];
            contravariant(Ja, F, G, ft2, gt2);
#pragma unroll
            for (int v = 0; v < NV; ++v) { F[v] = ft2[v]; G[v] = gt2[v]; }
        }
        store_traces<n>(a, e, i, j, U, F, G);
        line_put<N, C>(X, Y, el, i, j, F, G);
        if (SC) {
            double un[NV];
            load4w(a.u_base + ((size_t)e * nn + node) * NV, un);
            if constexpr (CURVED) sc_faces_curved<N, C, REC>(a, UU, VC, UF, FVX, FVY, el, e, i, j, un, blended, muscl, fx, fy);
            else sc_faces<N, C>(a, UU, VC, FVX, FVY, el, e, i, j, un, blended, fx, fy);
        }
    }
    phase_sync<C>();
    line_contract<N, C, true>(X, Y, tid);
    phase_sync<C>();
    // the step's final values: per-element CFL slots as the LW kernel writes them (plain TreeMesh MDRK step)
    constexpr bool SLOTS = MODE == MODE_STEP && !SC;
    double l1 = 0.0, l2 = 0.0;
    if (active) {
        double acc[NV];
        node_sum<N, C>(X, Y, el, i, j, acc);
        if (SC) {
            if constexpr (CURVED) sc_blend_curved<N, C>(FVX, FVY, el, i, j, alpha_e, blended, fx, fy, acc);
            else if (blended) sc_blend<N, C>(FVX, FVY, el, i, j, alpha_e, fx, fy, acc);
        }
        double o[NV], ub[NV];
        if (MODE == MODE_STEP) load4w(a.u_base + ((size_t)e * nn + node) * NV, ub);
        store_result<MODE>(a.out + ((size_t)e * nn + node) * NV, MODE == MODE_STEP ? -dt * ij : -ij, dt, acc, ub,
                           SRC ? Ssrc : nullptr, o);
        if (SLOTS && a.cfl_slots && i > 0 && i < n - 1 && j > 0 && j < n - 1) {
            node_speeds(a.gamma, o, a.speed_status, l1, l2);
            if (CURVED) {
                const size_t k = (size_t)e * nn + node;
                double Jn[4];
                load4w_const(a.metrics + k * 4, Jn);
                curved_speeds(Jn, __ldg(a.inv_jac_node + k), l1, l2);
            }
        }
    }
    if (SLOTS && a.cfl_slots) write_interior_slots<N, C>(a, X, active, el, i, j, tid, l1, l2);
}

}  // namespace tlw
