// mps_stages.cu -- explicit per-particle stages of one MPS step (FP64).
//
// Each particle's neighbour row is walked by a group of lanes.  Every
// support / cutoff decision the reference takes with sqrt() is taken here on
// the squared distance against an exact threshold (same decision, see
// sqrt_cut), and magnitudes use one rsqrt per pair instead of the
// reference's sqrt and four divisions (functions.cu:32-89, 245-428), so each
// term differs from the reference's by a few ulps at most.  Positions and
// velocities are gathered as packed double4.  Lists are row-major (see
// mps_internal.cuh): a group of G lanes walks one row, entries k = lane,
// lane + G, ..., and the group's partial sums meet in a fixed butterfly.
// Reference routines are cited on each kernel.
#include "mps_internal.cuh"

using namespace vmps;

namespace {

struct Lists {
    const int* __restrict__ nbr;
    const int* __restrict__ len;
    int cap;
};

__device__ __forceinline__ const int* row_of(const Lists& L, int i)
{
    return L.nbr + (size_t)i * L.cap;
}

template <int DIM>
__device__ __forceinline__ double d2of(const double4& a, const double4& b, double& dx, double& dy,
                                       double& dz)
{
    dx = b.x - a.x;
    dy = b.y - a.y;
    dz = DIM == 3 ? b.z - a.z : 0.0;
    return dist2<DIM>(dx, dy, dz);
}

// positions (x, y, z, ptype) when ptype != nullptr, else (a, b, c, 0)
__global__ void k_pack(int n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ z, const int* __restrict__ ptype,
                       double4* __restrict__ P4)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) P4[i] = make_double4(x[i], y[i], z[i], ptype ? (double)ptype[i] : 0.0);
}

// BCON's class of a particle (functions.cu:433-445)
__device__ __forceinline__ int bcon_of(int ptype, double nd, double n0, double dirichlet)
{
    if (ptype <= -1) return -1;
    return nd / n0 < dirichlet ? 1 : 0;
}

// BCON in PNUMSTAR's pass (bcon null: PNUM or PNUMSTAR alone)
struct BconOut {
    int* bcon;
    const int* ptype;
    double n0, dirichlet;
};

// PNUM / PNUMSTAR (functions.cu:94-122, 157-179)
template <int DIM, int G, int KT>
__global__ void __launch_bounds__(256, 8) k_pnd(int n, Lists L, const double4* __restrict__ P4, WK wk, int correct,
                      double ncorr, double* __restrict__ out, unsigned long long* dmax, BconOut B)
{
    Grp<G> q;
    int i = (int)q.gid;
    if (i >= n) return;
    double4 pi = P4[i];
    const int* row = row_of(L, i);
    int len = L.len[i];
    double sum = 0.0;
    for (int k = q.lane; k < len; k += G) {
        int j = row[k];
        if (i == j) continue;
        double dx, dy, dz;
        double d2 = d2of<DIM>(pi, ld4(P4 + j), dx, dy, dz);
        sum += w_fast<DIM, KT>(wk, d2, rsq(d2));
    }
    sum = q.sum(sum);
    if (q.lane == 0) {
        if (correct && wk.ktype != 2) sum = sum * ncorr;
        out[i] = sum;
        if (B.bcon) B.bcon[i] = bcon_of(B.ptype[i], sum, B.n0, B.dirichlet);
        // non-negative doubles order as their bit patterns
        if (dmax && sum > 0.0) atomicMax(dmax, (unsigned long long)__double_as_longlong(sum));
    }
}

// The start of a step's explicit stages in one launch: the packed positions with
// the previous pressure that PREDICTION gathers, and, where they need no
// neighbours, V_FRACTION's C (no second fluid: zero) and VISCOSITY's meu (Newtonian
// fluids: by kind).  C and meu are null when their own stages run.
__global__ void k_explicit_begin(int n, const double* __restrict__ x,
                                 const double* __restrict__ y, const double* __restrict__ z,
                                 const double* __restrict__ pnew, const int* __restrict__ ptype, double meu1, double meu2,
                                 double4* __restrict__ PP4, double* __restrict__ C,
                                 double* __restrict__ meu)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    PP4[i] = make_double4(x[i], y[i], z[i], pnew[i]);
    if (C) C[i] = 0.0;
    if (meu) {
        const int pt = ptype[i];
        if (pt <= 1) meu[i] = meu1;
        if (pt == 2) meu[i] = meu2;
    }
}

// BCON (functions.cu:433-445)
// P4w (the predicted positions the PPE is assembled at, or null): its w
// slot, unread after PNUMSTAR, takes bcon so that the assembly finds each
// neighbour's position and status in one gather
__global__ void k_bcon(int n, const int* __restrict__ ptype, const double* __restrict__ nd,
                       double n0, double dirichlet, int* __restrict__ bcon,
                       double4* __restrict__ P4w)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = bcon_of(ptype[i], nd[i], n0, dirichlet);
    bcon[i] = b;
    if (P4w) reinterpret_cast<double*>(P4w + i)[3] = (double)b;
}

// V_FRACTION (functions.cu:2580-2638)
template <int DIM, int G, int KT>
__global__ void k_vfraction(int n, Lists L, const int* __restrict__ ptype,
                            const double4* __restrict__ P4, WK wk, int method,
                            double* __restrict__ C)
{
    Grp<G> q;
    int I = (int)q.gid;
    if (I >= n) return;
    double sum1 = 0, sum2 = 0;
    double4 pi = P4[I];
    const int* row = row_of(L, I);
    int len = L.len[I];
    for (int k = q.lane; k < len; k += G) {
        int J = row[k];
        int pj = ptype[J];
        if (I == J || pj <= 0) continue;
        double w = 1.0;
        if (method != 1) {
            double dx, dy, dz;
            double d2 = d2of<DIM>(pi, ld4(P4 + J), dx, dy, dz);
            w = w_fast<DIM, KT>(wk, d2, rsq(d2));
        }
        sum1 += w;
        if (pj == 2) sum2 += w;
    }
    sum1 = q.sum(sum1);
    sum2 = q.sum(sum2);
    if (q.lane == 0) {
        double c = sum2 / sum1;
        if (sum1 == 0) c = 0;
        C[I] = c;
    }
}

// velocity-gradient sums of VISCOSITY / SPS (functions.cu:2096-2117, 1734-1756);
// mind2 < 0: every pair (VISCOSITY); else pairs with d2 > mind2 (SPS d > coll/10).
// Returns the group-reduced sums in every lane.
template <int DIM, int G, int KT>
__device__ __forceinline__ void grad_sums(const Grp<G>& q, const Lists& L, int I,
                                          const double4* P4, const double* un, const double* vn,
                                          const double* wn, const WK& wk, double mind2, double* s)
{
    for (int k = 0; k < 9; k++) s[k] = 0.0;
    const int* row = row_of(L, I);
    int len = L.len[I];
    double4 pi = P4[I];
    double ui = un[I], vi = vn[I], wi = DIM == 3 ? wn[I] : 0.0;
    for (int k = q.lane; k < len; k += G) {
        int j = row[k];
        if (I == j) continue;
        double dx, dy, dz;
        double d2 = d2of<DIM>(pi, ld4(P4 + j), dx, dy, dz);
        if (!(mind2 < 0 || d2 > mind2)) continue;
        double rD = rsq(d2);
        double f = w_fast<DIM, KT>(wk, d2, rD) * rD * rD;
        double du = un[j] - ui, dv = vn[j] - vi;
        s[0] += du * dx * f;
        s[1] += dv * dy * f;
        s[2] += du * dy * f;
        s[3] += dv * dx * f;
        if (DIM == 3) {
            double dw = wn[j] - wi;
            s[4] += dw * dz * f;
            s[5] += du * dz * f;
            s[6] += dv * dz * f;
            s[7] += dw * dx * f;
            s[8] += dw * dy * f;
        }
    }
    for (int k = 0; k < (DIM == 3 ? 9 : 4); k++) s[k] = q.sum(s[k]);
}

// strain tensor S11 S12 S22 S13 S23 S33 (functions.cu:2118-2146)
template <int DIM>
__device__ __forceinline__ void strain(double n0, const double* s, double* S)
{
    double Uxx = (2.0 / n0) * s[0], Uyy = (2.0 / n0) * s[1];
    double Uxy = (2.0 / n0) * s[2], Uyx = (2.0 / n0) * s[3];
    S[1] = 0.5 * (Uxy + Uyx);
    S[0] = 0.5 * (Uxx + Uxx);
    S[2] = 0.5 * (Uyy + Uyy);
    S[3] = S[4] = S[5] = 0.0;
    if (DIM == 3) {
        double Uzz = (2.0 / n0) * s[4], Uxz = (2.0 / n0) * s[5], Uyz = (2.0 / n0) * s[6];
        double Uzx = (2.0 / n0) * s[7], Uzy = (2.0 / n0) * s[8];
        S[5] = 0.5 * (Uzz + Uzz);
        S[3] = 0.5 * (Uxz + Uzx);
        S[4] = 0.5 * (Uyz + Uzy);
    }
}

struct Phys {
    double rho1, rho2, nu1, nu2, n0, meu0, n_pl, phi, cohes, cs, l0, mind2;
    int fluid2_type;
    WK wk;
};

// VISCOSITY (functions.cu:2053-2184); reads C[i] where the reference reads
// C[0] (identical whenever phi == 0)
template <int DIM, int G, int KT>
__global__ void k_viscosity(int n, Lists L, Phys P, const int* __restrict__ ptype,
                            const double4* __restrict__ P4, const double* __restrict__ un,
                            const double* __restrict__ vn, const double* __restrict__ wn,
                            const double* __restrict__ C, const double* __restrict__ phat,
                            double* __restrict__ meu)
{
    Grp<G> q;
    int i = (int)q.gid;
    if (i >= n) return;
    int pt = ptype[i];
    if (P.fluid2_type == 0) {
        if (q.lane == 0) {
            if (pt <= 1) meu[i] = P.nu1 * P.rho1;
            if (pt == 2) meu[i] = P.nu2 * P.rho2;
        }
        return;
    }
    if (pt == 1) {
        if (q.lane == 0) meu[i] = P.nu1 * P.rho1;
        return;
    }
    double s[9], S[6];
    grad_sums<DIM, G, KT>(q, L, i, P4, un, vn, wn, P.wk, -1.0, s);
    if (q.lane != 0) return;
    strain<DIM>(P.n0, s, S);
    double phi = (C[i] - 0.25) * P.phi / (1 - 0.25);
    if (C[i] < 0.25) phi = 0;
    double yield_stress = P.cohes * cos(phi) + phat[i] * sin(phi);
    double S11 = S[0], S12 = S[1], S22 = S[2], S13 = S[3], S23 = S[4], S33 = S[5];
    double II;
    if (DIM == 3)
        II = fabs((S11 * S22 * S33 + S12 * S23 * S13 + S13 * S12 * S23) -
                  (S13 * S22 * S13 + S11 * S23 * S23 + S12 * S12 * S33));
    else
        II = fabs(S11 * S22 - S12 * S12);
    double m = yield_stress / 2 / sqrt(II) + P.meu0 * pow(4 * II, (P.n_pl - 1) / 2);
    if (II == 0 || m > 200) m = 200;
    meu[i] = m;
}

// SPS pass 1: strain tensor and eddy viscosity (functions.cu:1731-1790)
template <int DIM, int G, int KT>
__global__ void k_sps1(int n, Lists L, Phys P, const int* __restrict__ ptype,
                       const double4* __restrict__ P4, const double* __restrict__ un,
                       const double* __restrict__ vn, const double* __restrict__ wn,
                       double* __restrict__ S6, double* __restrict__ neut)
{
    Grp<G> q;
    int i = (int)q.gid;
    if (i >= n || ptype[i] < 0) return;
    double s[9], S[6];
    grad_sums<DIM, G, KT>(q, L, i, P4, un, vn, wn, P.wk, P.mind2, s);
    if (q.lane != 0) return;
    strain<DIM>(P.n0, s, S);
    for (int c = 0; c < 6; c++) S6[(size_t)c * n + i] = S[c];
    double S11 = S[0], S12 = S[1], S22 = S[2], S13 = S[3], S23 = S[4], S33 = S[5];
    double Sm;
    if (DIM == 3)
        Sm = sqrt(2 * S11 * S11) + 2 * sqrt(2 * S12 * S12) + sqrt(2 * S22 * S22) +
             sqrt(2 * S33 * S33) + 2 * sqrt(2 * S13 * S13) + 2 * sqrt(2 * S23 * S23);
    else
        Sm = sqrt(2 * S11 * S11) + 2 * sqrt(2 * S12 * S12) + sqrt(2 * S22 * S22);
    double cd = P.cs * P.l0;
    neut[i] = (cd * cd) * Sm;
}

// SPS pass 2: divergence of the SPS stress (functions.cu:1793-1830)
template <int DIM, int G, int KT>
__global__ void k_sps2(int n, Lists L, Phys P, const int* __restrict__ ptype,
                       const double4* __restrict__ P4, const double* __restrict__ S6,
                       const double* __restrict__ neut, double* __restrict__ t1,
                       double* __restrict__ t2, double* __restrict__ t3)
{
    Grp<G> q;
    int i = (int)q.gid;
    if (i >= n || ptype[i] < 0) return;
    double sum1 = 0, sum2 = 0, sum3 = 0;
    const int* row = row_of(L, i);
    int len = L.len[i];
    double ni = neut[i];
    double4 pi = P4[i];
    for (int k = q.lane; k < len; k += G) {
        int j = row[k];
        if (i == j) continue;
        double dx, dy, dz;
        double d2 = d2of<DIM>(pi, ld4(P4 + j), dx, dy, dz);
        if (!(d2 > P.mind2)) continue;
        double rD = rsq(d2);
        double f = (neut[j] - ni) * w_fast<DIM, KT>(P.wk, d2, rD) * rD * rD;
        sum1 += dx * f;
        sum2 += dy * f;
        if (DIM == 3) sum3 += dz * f;
    }
    sum1 = q.sum(sum1);
    sum2 = q.sum(sum2);
    sum3 = q.sum(sum3);
    if (q.lane != 0) return;
    double S11 = S6[i], S12 = S6[(size_t)n + i], S22 = S6[2 * (size_t)n + i];
    double S13 = S6[3 * (size_t)n + i], S23 = S6[4 * (size_t)n + i], S33 = S6[5 * (size_t)n + i];
    if (DIM == 3) {
        t1[i] = (2.0 / P.n0) * (2 * S11 * sum1 + 2 * S12 * sum2 + 2 * S13 * sum3);
        t2[i] = (2.0 / P.n0) * (2 * S12 * sum1 + 2 * S22 * sum2 + 2 * S23 * sum3);
        t3[i] = (2.0 / P.n0) * (2 * S13 * sum1 + 2 * S23 * sum2 + 2 * S33 * sum3);
    } else {
        t1[i] = (2.0 / P.n0) * (2 * S11 * sum1 + 2 * S12 * sum2);
        t2[i] = (2.0 / P.n0) * (2 * S12 * sum1 + 2 * S22 * sum2);
    }
}

struct PredArgs {
    WK ws, wl;
    double n0_s, visc_coef, dt, gx, gy, gz, relaxp, rho1, rho2;
    // Newtonian fluids (BYKIND): VISCOSITY sets meu by particle kind (nu1 rho1
    // for kinds <= 1, nu2 rho2 for kind 2), so a pair's viscosity follows from
    // the two kinds, without a gather of meu and with the two divisions of the
    // mixed value made once per particle
    double meu1, meu2;
};

// PREDICTION (functions.cu:2283-2369), first part: the explicit pressure
// sums over the PND list, scaled by (1-relaxp)*2*dt/(n0*rho) (fluid rows).
// Bound by the L1's sector rate, as the other sums over the PND list; 6
// resident blocks per SM (476 k-particle dam: 79 us, 82 us at 5 blocks, 99 us
// with 128-bit gathers and the general kernel function)
template <int DIM, int G, int KT>
__global__ void __launch_bounds__(256, 6) k_predict_p(int n, Lists Ls, PredArgs A, const double4* __restrict__ P4,
                            const double4* __restrict__ PP4, const double* __restrict__ phat,
                            const double* __restrict__ rho, double* __restrict__ px,
                            double* __restrict__ py, double* __restrict__ pz)
{
    Grp<G> q;
    int I = (int)q.gid;
    if (I >= n) return;
    if (P4[I].w <= 0) return;
    const double4 pi = PP4[I];
    double sum1 = 0, sum2 = 0, sum3 = 0;
    double ph = phat[I];
    const int* row = row_of(Ls, I);
    int len = Ls.len[I];
    for (int k = q.lane; k < len; k += G) {
        int J = row[k];
        if (I == J) continue;
        double dx, dy, dz;
        const double4 pj = ld4(PP4 + J);  // position and previous pressure in one gather
        double d2 = d2of<DIM>(pi, pj, dx, dy, dz);
        if (!(d2 > 0)) continue;
        double rD = rsq(d2);
        double f = (pj.w - ph) * w_fast<DIM, KT>(A.ws, d2, rD) * rD * rD;
        sum1 += dx * f;
        sum2 += dy * f;
        if (DIM == 3) sum3 += dz * f;
    }
    sum1 = q.sum(sum1);
    sum2 = q.sum(sum2);
    if (DIM == 3) sum3 = q.sum(sum3);
    if (q.lane != 0) return;
    double pc = (1 - A.relaxp) * (2.0 * A.dt / A.n0_s / rho[I]);
    px[I] = pc * sum1;
    py[I] = pc * sum2;
    if (DIM == 3) pz[I] = pc * sum3;
}

// lanes per particle of the FP32 viscous sums (explicit stages of the 1.6 M-particle
// dam: 4 lanes 1.97 ms, 8 1.99, 16 2.17, a warp 2.48)
constexpr int kPred32G = 8;
// Mixed precision: the viscous Laplacian's neighbour sums in FP32 (FP32
// positions relative to the box, FP32 velocities, FP32 weights and sums);
// u* and x* are then formed in FP64 exactly as in k_predict.
// TURB: the eddy-viscosity sums (sum7..9, times neut) are kept only with
// SPS on; without it neut is 0 and they add nothing.
template <int DIM, bool TURB, int KT, bool BYKIND>
// 4 blocks per SM, which the general kernel function's registers once needed; with its
// type known at compile time 5 blocks measure better (explicit stages of the 1.6 M dam
// 1.99 ms at 4, 1.73 ms at 5)
__global__ void __launch_bounds__(256, 4)
k_predict32(int n, Lists Ll, PredArgs A, WKf wl, const double* __restrict__ meu,
            const double4* __restrict__ P4, const double4* __restrict__ U4,
            const float4* __restrict__ P4f, const float4* __restrict__ U4f,
            const double* __restrict__ px, const double* __restrict__ py,
            const double* __restrict__ pz, const double* __restrict__ neut,
            const double* __restrict__ t1, const double* __restrict__ t2,
            const double* __restrict__ t3, double* __restrict__ xs, double* __restrict__ ys,
            double* __restrict__ zs, double* __restrict__ us, double* __restrict__ vs,
            double* __restrict__ ws, double4* __restrict__ P4s, float4* __restrict__ P4sf,
            double3 box0)
{
    Grp<kPred32G> q;
    int I = (int)q.gid;
    if (I >= n) return;
    double4 pi = P4[I], ui4 = U4[I];
    int pI = (int)pi.w;
    // precision 2: the predicted positions in FP32 too, relative to the box
    auto put_f = [&](const double4& o) {
        if (P4sf)
            P4sf[I] = make_float4((float)(o.x - box0.x), (float)(o.y - box0.y),
                                  DIM == 3 ? (float)(o.z - box0.z) : 0.f, o.w);
    };
    if (pI <= 0) {
        if (q.lane == 0) {
            xs[I] = pi.x; ys[I] = pi.y; us[I] = ui4.x; vs[I] = ui4.y;
            if (DIM == 3) { zs[I] = pi.z; ws[I] = ui4.z; }
            P4s[I] = pi;
            put_f(pi);
        }
        return;
    }
    const float4 fi = P4f[I], vi = U4f[I];
    float s4 = 0.f, s5 = 0.f, s6 = 0.f, s7 = 0.f, s8 = 0.f, s9 = 0.f;
    const double mI = meu[I];
    const double rhoI = (pI == 1) ? A.rho1 : A.rho2;
    const float neu_same = (float)(mI / rhoI);
    auto mixed = [&](double mJ) { return 2 * mI * mJ / (mI + mJ) / rhoI; };
    const float neu_1 = BYKIND ? (float)mixed(A.meu1) : 0.f;
    const float neu_2 = BYKIND ? (float)mixed(A.meu2) : 0.f;
    const int* row = row_of(Ll, I);
    int len = Ll.len[I];
    auto add = [&](int J, const float4& fj, const float4& vj) {
        if (I == J) return;
        const float dx = fj.x - fi.x, dy = fj.y - fi.y, dz = DIM == 3 ? fj.z - fi.z : 0.f;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        if (!(d2 > 0.f)) return;
        const float W = w_fast32<DIM, KT>(wl, d2);
        float NEU = neu_same;
        if ((int)fj.w != pI) {
            if (BYKIND) NEU = (int)fj.w == 2 ? neu_2 : neu_1;
            else NEU = (float)mixed(meu[J]);
        }
        const float du = W * (vj.x - vi.x), dv = W * (vj.y - vi.y);
        s4 = __fmaf_rn(du, NEU, s4);
        s5 = __fmaf_rn(dv, NEU, s5);
        if (TURB) {
            s7 += du;
            s8 += dv;
        }
        if (DIM == 3) {
            const float dw = W * (vj.z - vi.z);
            s6 = __fmaf_rn(dw, NEU, s6);
            if (TURB) s9 += dw;
        }
    };
    // two entries per lane in flight (k, k + G); the sums see them in list order
    for (int k = q.lane; k < len; k += 2 * kPred32G) {
        const bool two = k + kPred32G < len;
        const int J0 = row[k], J1 = two ? row[k + kPred32G] : I;
        const float4 f0 = P4f[J0], f1 = P4f[J1], v0 = U4f[J0], v1 = U4f[J1];
        add(J0, f0, v0);
        add(J1, f1, v1);
    }
    double sum4 = q.sum((double)s4), sum5 = q.sum((double)s5), sum7 = 0, sum8 = 0, sum6 = 0,
           sum9 = 0;
    if (TURB) { sum7 = q.sum((double)s7); sum8 = q.sum((double)s8); }
    if (DIM == 3) sum6 = q.sum((double)s6);
    if (DIM == 3 && TURB) sum9 = q.sum((double)s9);
    if (q.lane != 0) return;
    double DT = A.dt, nt = TURB ? neut[I] : 0.0;
    double uS = ui4.x + A.gx * DT + A.visc_coef * (sum4 + nt * sum7) + DT * t1[I] - px[I];
    double vS = ui4.y + A.gy * DT + A.visc_coef * (sum5 + nt * sum8) + DT * t2[I] - py[I];
    double4 o = pi;
    o.x = pi.x + DT * uS;
    o.y = pi.y + DT * vS;
    us[I] = uS;
    vs[I] = vS;
    xs[I] = o.x;
    ys[I] = o.y;
    if (DIM == 3) {
        double wS = ui4.z + A.gz * DT + A.visc_coef * (sum6 + nt * sum9) + DT * t3[I] - pz[I];
        ws[I] = wS;
        o.z = pi.z + DT * wS;
        zs[I] = o.z;
    }
    P4s[I] = o;
    put_f(o);
}

// PREDICTION, second part: viscous Laplacian over the Laplacian list, one
// group of kPredG lanes per particle, then u* and x*.
// lanes per particle of the viscous sums: 8 (explicit stages of the 1.6 M-particle
// dam: 4 lanes 2.60 ms, 8 2.54, 16 2.64, a warp 2.92)
// 128 threads at 72 registers (7 blocks, 28 warps per SM): the two entries in
// flight need them (256 threads at 64 registers spill: 507 against 497 us)
constexpr int kPredThreads = 128;
constexpr int kPredG = 8;
// TURB: the eddy-viscosity sums (sum7..9, times neut) are kept only with
// SPS on; without it neut is 0 and they add nothing.
// Bound by the L1 (77% of its throughput, 2 x 32 bytes gathered per entry).
// One 256-bit load per gathered vector, the kernel function's type known at
// compile time (its general form spills), two entries of a lane in flight:
// 497 us on the 476 k-particle dam against 652 us for 128-bit halves one
// entry at a time; larger blocks for L1 reuse (448 to 1024 threads) 518-559
// us, the next entry's index alone read ahead 543 us
template <int DIM, bool TURB, int KT, bool BYKIND>
__global__ void __launch_bounds__(kPredThreads, 7)
k_predict(int n, Lists Ll, PredArgs A, const double* __restrict__ meu,
          const double4* __restrict__ P4, const double4* __restrict__ U4,
          const double* __restrict__ px, const double* __restrict__ py,
          const double* __restrict__ pz, const double* __restrict__ neut,
          const double* __restrict__ t1, const double* __restrict__ t2,
          const double* __restrict__ t3, double* __restrict__ xs, double* __restrict__ ys,
          double* __restrict__ zs, double* __restrict__ us, double* __restrict__ vs,
          double* __restrict__ ws, double4* __restrict__ P4s)
{
    Grp<kPredG> q;
    int I = (int)q.gid;
    if (I >= n) return;
    double4 pi = P4[I], ui4 = U4[I];
    int pI = (int)pi.w;
    if (pI <= 0) {
        if (q.lane == 0) {
            xs[I] = pi.x; ys[I] = pi.y; us[I] = ui4.x; vs[I] = ui4.y;
            if (DIM == 3) { zs[I] = pi.z; ws[I] = ui4.z; }
            P4s[I] = pi;
        }
        return;
    }
    double sum4 = 0, sum5 = 0, sum6 = 0, sum7 = 0, sum8 = 0, sum9 = 0;
    double mI = meu[I];
    double rhoI = (pI == 1) ? A.rho1 : A.rho2;
    double neu_same = mI / rhoI;
    auto mixed = [&](double mJ) { return 2 * mI * mJ / (mI + mJ) / rhoI; };
    const double neu_1 = BYKIND ? mixed(A.meu1) : 0.0, neu_2 = BYKIND ? mixed(A.meu2) : 0.0;
    const int* row = row_of(Ll, I);
    int len = Ll.len[I];
    auto add = [&](int J, const double4& pj, const double4& uj) {
        if (I == J) return;
        double dx, dy, dz;
        double d2 = d2of<DIM>(pi, pj, dx, dy, dz);
        if (!(d2 > 0)) return;
        double W = w_fast<DIM, KT>(A.wl, d2, rsq(d2));
        double NEU = neu_same;
        if ((int)pj.w != pI) {
            if (BYKIND) NEU = (int)pj.w == 2 ? neu_2 : neu_1;
            else NEU = mixed(meu[J]);
        }
        double du = W * (uj.x - ui4.x), dv = W * (uj.y - ui4.y);
        sum4 += du * NEU;
        sum5 += dv * NEU;
        if (TURB) {
            sum7 += du;
            sum8 += dv;
        }
        if (DIM == 3) {
            double dw = W * (uj.z - ui4.z);
            sum6 += dw * NEU;
            if (TURB) sum9 += dw;
        }
    };
    // two entries per lane in flight (k, k + G); the sums see them in list order
    for (int k = q.lane; k < len; k += 2 * kPredG) {
        const int J0 = row[k], J1 = k + kPredG < len ? row[k + kPredG] : I;
        const double4 p0 = ld4(P4 + J0), p1 = ld4(P4 + J1), u0 = ld4(U4 + J0), u1 = ld4(U4 + J1);
        add(J0, p0, u0);
        add(J1, p1, u1);
    }
    sum4 = q.sum(sum4); sum5 = q.sum(sum5);
    if (TURB) { sum7 = q.sum(sum7); sum8 = q.sum(sum8); }
    if (DIM == 3) sum6 = q.sum(sum6);
    if (DIM == 3 && TURB) sum9 = q.sum(sum9);
    if (q.lane != 0) return;
    // read again rather than kept through the loop (registers)
    pi = ld4_again(P4 + I);
    ui4 = ld4_again(U4 + I);
    double DT = A.dt, nt = TURB ? neut[I] : 0.0;
    double uS = ui4.x + A.gx * DT + A.visc_coef * (sum4 + nt * sum7) + DT * t1[I] - px[I];
    double vS = ui4.y + A.gy * DT + A.visc_coef * (sum5 + nt * sum8) + DT * t2[I] - py[I];
    double4 o = pi;
    o.x = pi.x + DT * uS;
    o.y = pi.y + DT * vS;
    us[I] = uS;
    vs[I] = vS;
    xs[I] = o.x;
    ys[I] = o.y;
    if (DIM == 3) {
        double wS = ui4.z + A.gz * DT + A.visc_coef * (sum6 + nt * sum9) + DT * t3[I] - pz[I];
        ws[I] = wS;
        o.z = pi.z + DT * wS;
        zs[I] = o.z;
    }
    P4s[I] = o;
}

// weakly compressible EOS (functions.cu:2467-2500)
__global__ void k_pressure_wc(int n, const int* __restrict__ ptype, const double* __restrict__ C,
                              const double* __restrict__ nstar, double n0, double beta, double c01,
                              double c02, double rho1, double rho2, double pmin, double pmax,
                              double* __restrict__ pnew)
{
    int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= n || ptype[I] < 0) return;
    double c0 = (ptype[I] == 2) ? c02 : c01;
    double Rho = rho2 * C[I] + rho1 * (1 - C[I]);
    double p;
    if (nstar[I] < beta * n0) p = 0.0;
    else p = (c0 * c0 * Rho / 7.0) * (pow(nstar[I] / n0, 7.0) - 1);
    if (p < pmin) p = pmin;
    if (p > pmax) p = pmax;
    pnew[I] = p;
}

// PHATCALC (functions.cu:207-224); also packs (pnew, phat) for the gradient
template <int G>
__global__ void k_phat(int n, Lists L, const double* __restrict__ pnew, double* __restrict__ phat,
                       double2* __restrict__ PH, float2* __restrict__ PH32)
{
    Grp<G> q;
    int I = (int)q.gid;
    if (I >= n) return;
    double mn = 999999999999999;
    const int* row = row_of(L, I);
    int len = L.len[I];
    for (int k = q.lane; k < len; k += G) {
        double pj = pnew[row[k]];
        if (pj < mn) mn = pj;
    }
    mn = q.min(mn);
    if (q.lane == 0) {
        phat[I] = mn;
        PH[I] = make_double2(pnew[I], mn);
        if (PH32) PH32[I] = make_float2((float)pnew[I], (float)mn);
    }
}

struct Box {
    double xmin, xmax, ymin, ymax, zmin, zmax, dl, dt, cc;
    const int* scene;     // per-particle scene, or nullptr for one scene
    const double* sbox;   // 6 per scene
};

// the box of particle I: its scene's when scenes are batched
__device__ __forceinline__ void box_of(const Box& B, int I, double* b)
{
    if (B.scene) {
        const double* q = B.sbox + 6 * B.scene[I];
        for (int k = 0; k < 6; k++) b[k] = q[k];
    } else {
        b[0] = B.xmin; b[1] = B.xmax; b[2] = B.ymin; b[3] = B.ymax; b[4] = B.zmin; b[5] = B.zmax;
    }
}

// EULERINTEGRATION + BOUNDARIE (functions.cu:1963-2021) of one particle that
// moves with (ui, vi, wi)
template <int DIM>
__device__ __forceinline__ void move_particle(const Box& B, int I, double ui, double vi, double wi,
                                              double* __restrict__ x, double* __restrict__ y,
                                              double* __restrict__ z, double* __restrict__ un,
                                              double* __restrict__ vn, double* __restrict__ wn,
                                              double4* __restrict__ P4)
{
    double DT = B.dt, DL = B.dl, CC = B.cc;
    double bx[6];
    box_of(B, I, bx);
    double xi = x[I] + ui * DT, yi = y[I] + vi * DT;
    if (yi < bx[2] + DL * 3.0) { vi = fabs(vi) * CC; yi = bx[2] + DL * 3.0; }
    if (yi > bx[3] - DL * 3.0) { vi = -fabs(vi) * CC; yi = bx[3] - DL * 3.0; }
    if (xi < bx[0] + DL * 3.0) { ui = fabs(ui) * CC; xi = bx[0] + DL * 3.0; }
    if (xi > bx[1] - DL * 3.0) { ui = -fabs(ui) * CC; xi = bx[1] - DL * 3.0; }
    double zi = 0.0;
    if (DIM == 3) {
        zi = z[I] + wi * DT;
        if (zi < bx[4] + DL * 3.0) { wi = fabs(wi) * CC; zi = bx[4] + DL * 3.0; }
        if (zi > bx[5] - DL * 3.0) { wi = -fabs(wi) * CC; zi = bx[5] - DL * 3.0; }
        z[I] = zi;
        wn[I] = wi;
    }
    x[I] = xi; y[I] = yi; un[I] = ui; vn[I] = vi;
    P4[I] = make_double4(xi, yi, zi, P4[I].w);
}

// the arrays EULERINTEGRATION moves, for PRESSGRAD's pass
struct MoveArgs {
    Box B;
    double *x, *y, *z;
    double4* P4;
};

struct GradArgs {
    WK wk;
    double coef, vmax;
    int kh;
};

// PRESSGRAD (functions.cu:245-355), CPU semantics (p^_i + p^_j); MOVE: and
// EULERINTEGRATION of the particle with its new velocity
// 6 resident blocks per SM (40 registers): 101 us on the 476 k-particle dam, 104
// us at 5
template <int DIM, int G, int KT, bool MOVE>
__global__ void __launch_bounds__(256, 6) k_pressgrad(int n, Lists L, GradArgs A, const int* __restrict__ ptype,
                            const double2* __restrict__ PH, const double4* __restrict__ P4s,
                            const double* __restrict__ rho, const double* __restrict__ us,
                            const double* __restrict__ vs, const double* __restrict__ ws,
                            double* __restrict__ un, double* __restrict__ vn,
                            double* __restrict__ wn, MoveArgs M)
{
    Grp<G> q;
    int I = (int)q.gid;
    if (I >= n || ptype[I] <= 0) return;
    double sum1 = 0, sum2 = 0, sum3 = 0;
    double4 pi = P4s[I];
    double2 phI = PH[I];
    const int* row = row_of(L, I);
    int len = L.len[I];
    for (int k = q.lane; k < len; k += G) {
        int J = row[k];
        if (I == J) continue;
        double dx, dy, dz;
        double d2 = d2of<DIM>(pi, ld4(P4s + J), dx, dy, dz);
        double rD = rsq(d2);
        double2 phJ = PH[J];
        double pp = (A.kh == 1) ? phJ.x + phI.x - (phI.y + phJ.y) : phJ.x - phI.y;
        double f = pp * w_fast<DIM, KT>(A.wk, d2, rD) * rD * rD;
        sum1 += dx * f;
        sum2 += dy * f;
        if (DIM == 3) sum3 += dz * f;
    }
    sum1 = q.sum(sum1);
    sum2 = q.sum(sum2);
    if (DIM == 3) sum3 = q.sum(sum3);
    if (q.lane != 0) return;
    double c = A.coef / rho[I], VMAX = A.vmax, coeff = 2.0;
    double uN = us[I] - c * sum1;
    double vN = vs[I] - c * sum2;
    if (fabs(uN) > coeff * VMAX) uN = VMAX;
    if (vN > coeff * VMAX) vN = coeff * VMAX;
    if (vN < -coeff * VMAX) vN = -coeff * VMAX;
    double wN = 0.0;
    if (DIM == 3) {
        wN = ws[I] - c * sum3;
        if (fabs(wN) > coeff * VMAX) wN = VMAX;
    }
    if (MOVE) {
        move_particle<DIM>(M.B, I, uN, vN, wN, M.x, M.y, M.z, un, vn, wn, M.P4);
        return;
    }
    un[I] = uN;
    vn[I] = vN;
    if (DIM == 3) wn[I] = wN;
}

// Precision 2: PNUMSTAR (functions.cu:157-201) with FP32 positions relative
// to the box, FP32 weights and an FP32 sum; n* is stored in FP64 and the
// source (n* - n0) / n0 is formed from it in FP64.
template <int DIM, int G, int KT>
__global__ void k_pnd32(int n, Lists L, const float4* __restrict__ P4f, WKf wk,
                        double* __restrict__ out)
{
    Grp<G> q;
    int i = (int)q.gid;
    if (i >= n) return;
    const float4 pi = P4f[i];
    const int* row = row_of(L, i);
    int len = L.len[i];
    float sum = 0.f;
    for (int k = q.lane; k < len; k += G) {
        int j = row[k];
        if (i == j) continue;
        const float4 pj = P4f[j];
        const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = DIM == 3 ? pj.z - pi.z : 0.f;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        if (d2 > 0.f) sum += w_fast32<DIM, KT>(wk, d2);
    }
    sum = q.sumf(sum);
    if (q.lane == 0) out[i] = (double)sum;
}

// Precision 2: PRESSGRAD (functions.cu:245-355) with FP32 positions,
// pressures, weights and sums; u^{n+1} = u* - c * sum formed in FP64.
template <int DIM, int G, int KT>
__global__ void __launch_bounds__(256, 5) k_pressgrad32(int n, Lists L, GradArgs A, WKf wk,
                            const int* __restrict__ ptype, const float2* __restrict__ PH32,
                            const float4* __restrict__ P4sf, const double* __restrict__ rho,
                            const double* __restrict__ us, const double* __restrict__ vs,
                            const double* __restrict__ ws, double* __restrict__ un,
                            double* __restrict__ vn, double* __restrict__ wn)
{
    Grp<G> q;
    int I = (int)q.gid;
    if (I >= n || ptype[I] <= 0) return;
    float s1 = 0.f, s2 = 0.f, s3 = 0.f;
    const float4 pi = P4sf[I];
    const float2 phI = PH32[I];
    const int* row = row_of(L, I);
    int len = L.len[I];
    for (int k = q.lane; k < len; k += G) {
        int J = row[k];
        if (I == J) continue;
        const float4 pj = P4sf[J];
        const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = DIM == 3 ? pj.z - pi.z : 0.f;
        const float d2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        if (!(d2 > 0.f)) continue;
        const float2 phJ = PH32[J];
        const float pp = (A.kh == 1) ? phJ.x + phI.x - (phI.y + phJ.y) : phJ.x - phI.y;
        const float f = pp * w_fast32<DIM, KT>(wk, d2) / d2;
        s1 = __fmaf_rn(dx, f, s1);
        s2 = __fmaf_rn(dy, f, s2);
        if (DIM == 3) s3 = __fmaf_rn(dz, f, s3);
    }
    const double sum1 = q.sum((double)s1), sum2 = q.sum((double)s2);
    const double sum3 = DIM == 3 ? q.sum((double)s3) : 0.0;
    if (q.lane != 0) return;
    double c = A.coef / rho[I], VMAX = A.vmax, coeff = 2.0;
    double uN = us[I] - c * sum1;
    double vN = vs[I] - c * sum2;
    if (fabs(uN) > coeff * VMAX) uN = VMAX;
    if (vN > coeff * VMAX) vN = coeff * VMAX;
    if (vN < -coeff * VMAX) vN = -coeff * VMAX;
    un[I] = uN;
    vn[I] = vN;
    if (DIM == 3) {
        double wN = ws[I] - c * sum3;
        if (fabs(wN) > coeff * VMAX) wN = VMAX;
        wn[I] = wN;
    }
}

// EULERINTEGRATION + BOUNDARIE (functions.cu:1963-2021)
template <int DIM>
__global__ void k_integrate(int n, Box B, const int* __restrict__ ptype, double* __restrict__ x,
                            double* __restrict__ y, double* __restrict__ z,
                            double* __restrict__ un, double* __restrict__ vn,
                            double* __restrict__ wn, double4* __restrict__ P4)
{
    int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= n || ptype[I] <= 0) return;
    move_particle<DIM>(B, I, un[I], vn[I], DIM == 3 ? wn[I] : 0.0, x, y, z, un, vn, wn, P4);
}

struct CollArgs {
    double coll2, cc, dt, rho1, rho2;
};

// One visit of COLLISION2's pair loop (functions.cu:1536-1599) from i's list
// to its neighbour j, on register copies s = {u, v, w, x, y, z} of the two
// states: the reference's expressions in the reference's order.
template <int DIM>
__device__ __forceinline__ void coll_visit(const CollArgs& A, int pti, int ptj, double* si,
                                           double* sj)
{
    const double m1 = (pti == 1) ? A.rho1 : A.rho2, m2 = (ptj == 1) ? A.rho1 : A.rho2;
    const double ex = sj[3] - si[3], ey = sj[4] - si[4], ez = DIM == 3 ? sj[5] - si[5] : 0.0;
    const double d2 = dist2<DIM>(ex, ey, ez);
    if (!(d2 < A.coll2)) return;
    const double d = sqrt(d2);
    const double ug = (m1 * si[0] + m2 * sj[0]) / (m1 + m2);
    const double vg = (m1 * si[1] + m2 * sj[1]) / (m1 + m2);
    const double ur = m1 * (si[0] - ug), vr = m1 * (si[1] - vg);
    double vabs;
    if (DIM == 3) {
        const double wg = (m1 * si[2] + m2 * sj[2]) / (m1 + m2);
        const double wr = m1 * (si[2] - wg);
        vabs = (ur * ex + vr * ey + wr * ez) / d;
    } else {
        vabs = (ur * ex + vr * ey) / d;
    }
    if (!(vabs > 0)) return;
    const double um = (1.0 + A.cc) * vabs * ex / d;
    const double vm = (1.0 + A.cc) * vabs * ey / d;
    const double wm = DIM == 3 ? (1.0 + A.cc) * vabs * ez / d : 0.0;
    if (pti > 0) {
        si[0] = si[0] - um / m1; si[1] = si[1] - vm / m1;
        si[3] = si[3] - A.dt * um / m1; si[4] = si[4] - A.dt * vm / m1;
        if (DIM == 3) { si[2] = si[2] - wm / m1; si[5] = si[5] - A.dt * wm / m1; }
    }
    if (ptj > 0) {
        sj[0] = sj[0] + um / m2; sj[1] = sj[1] + vm / m2;
        sj[3] = sj[3] + A.dt * um / m2; sj[4] = sj[4] + A.dt * vm / m2;
        if (DIM == 3) { sj[2] = sj[2] + wm / m2; sj[5] = sj[5] + A.dt * wm / m2; }
    }
}

// COLLISION2 (functions.cu:1523-1601) in an order-independent form.  The
// reference walks every particle, walls and dummies included, in id order
// and updates pairs in place, so a pair (a, b), a < b, is visited twice:
// from a's list, then from b's list with the state the first visit left (a
// fluid-wall pair can be pushed twice; a fluid-fluid pair separates after
// the first push).  Each fluid particle here replays, for every neighbour
// closer than coll in the pre-collision state, that pair's two visits in
// registers.  With one such neighbour the particle takes the replayed state
// -- COLLISION2's own result, bit for bit, as nothing else touches the pair
// in between; with several it takes the pre-collision state plus the sum of
// the pairs' changes.  The new states go to the *o arrays, and
// k_collision_apply copies them over once every particle has read the
// pre-collision state (no buffer swap, so the step's buffers stay fixed).
template <int DIM, int G>
__global__ void __launch_bounds__(256, 4) k_collision(int n, Lists L, CollArgs A, const int* __restrict__ ptype,
                            const int* __restrict__ oid, const double4* __restrict__ P4,
                            const double* __restrict__ un, const double* __restrict__ vn,
                            const double* __restrict__ wn, double* __restrict__ xo,
                            double* __restrict__ yo, double* __restrict__ zo,
                            double* __restrict__ uo, double* __restrict__ vo,
                            double* __restrict__ wo)
{
    Grp<G> q;
    const int i = (int)q.gid;
    if (i >= n) return;  // whole groups leave together
    const int pti = ptype[i];
    if (pti <= 0) return;
    const double4 pi = P4[i];
    const double s0[6] = {un[i], vn[i], DIM == 3 ? wn[i] : 0.0, pi.x, pi.y, DIM == 3 ? pi.z : 0.0};
    // the replay of pair (i, j) into si
    auto replay = [&](int j, const double4& pj, double* si) {
        double sj[6] = {un[j], vn[j], DIM == 3 ? wn[j] : 0.0, pj.x, pj.y, DIM == 3 ? pj.z : 0.0};
#pragma unroll
        for (int t = 0; t < 6; t++) si[t] = s0[t];
        const int ptj = ptype[j];
        if (oid[j] < oid[i]) {
            coll_visit<DIM>(A, ptj, pti, sj, si);
            coll_visit<DIM>(A, pti, ptj, si, sj);
        } else {
            coll_visit<DIM>(A, pti, ptj, si, sj);
            coll_visit<DIM>(A, ptj, pti, sj, si);
        }
    };
    // the hot loop only finds the neighbours closer than coll (rare); the
    // replays run after it
    int hits = 0, jhit = -1;
    const int* row = row_of(L, i);
    const int len = L.len[i];
    for (int k = q.lane; k < len; k += G) {
        const int j = row[k];
        if (i == j) continue;
        double ex, ey, ez;
        if (d2of<DIM>(pi, ld4(P4 + j), ex, ey, ez) < A.coll2) {
            hits++;
            jhit = j;
        }
    }
    int total = hits;
    for (int o = G / 2; o > 0; o >>= 1) total += __shfl_xor_sync(q.mask, total, o);
    double* const outs[6] = {uo, vo, wo, xo, yo, zo};
    if (total == 1) {  // the lane that met the one neighbour writes its replayed state
        if (hits == 1) {
            double si[6];
            replay(jhit, P4[jhit], si);
            for (int t = 0; t < 6; t++)
                if (DIM == 3 || (t != 2 && t != 5)) outs[t][i] = si[t];
        }
        return;
    }
    double acc[6] = {0, 0, 0, 0, 0, 0};
    if (total > 1) {  // several: the pre-collision state plus the sum of the replays' changes
        for (int k = q.lane; k < len; k += G) {
            const int j = row[k];
            if (i == j) continue;
            double ex, ey, ez;
            const double4 pj = P4[j];
            if (!(d2of<DIM>(pi, pj, ex, ey, ez) < A.coll2)) continue;
            double si[6];
            replay(j, pj, si);
#pragma unroll
            for (int t = 0; t < 6; t++) acc[t] += si[t] - s0[t];
        }
#pragma unroll
        for (int t = 0; t < 6; t++) acc[t] = q.sum(acc[t]);
    }
    if (q.lane != 0) return;
    for (int t = 0; t < 6; t++)
        if (DIM == 3 || (t != 2 && t != 5)) outs[t][i] = total > 1 ? s0[t] + acc[t] : s0[t];
}

template <int DIM>
__global__ void k_collision_apply(int n, const int* __restrict__ ptype, double* __restrict__ x,
                                  double* __restrict__ y, double* __restrict__ z,
                                  double* __restrict__ un, double* __restrict__ vn,
                                  double* __restrict__ wn, const double* __restrict__ xo,
                                  const double* __restrict__ yo, const double* __restrict__ zo,
                                  const double* __restrict__ uo, const double* __restrict__ vo,
                                  const double* __restrict__ wo, double4* __restrict__ P4)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || ptype[i] <= 0) return;
    double4 pi = P4[i];
    pi.x = xo[i];
    pi.y = yo[i];
    x[i] = pi.x;
    y[i] = pi.y;
    un[i] = uo[i];
    vn[i] = vo[i];
    if (DIM == 3) {
        pi.z = zo[i];
        z[i] = pi.z;
        wn[i] = wo[i];
    }
    P4[i] = pi;
}

// PREPDATA's ERROR#1 / ERROR#2 (functions.cu:2720-2743)
template <int DIM>
__device__ __forceinline__ void commit_checks(const Box& B, int I, double x, double y, double z,
                                              double u, double v, double w, double p,
                                              unsigned int* err)
{
    bool bad = p * 0 != 0 || u * 0 != 0 || v * 0 != 0 || (DIM == 3 && w * 0 != 0);
    double bx[6];
    box_of(B, I, bx);
    bool out = x >= bx[1] || y >= bx[3] || x <= bx[0] || y <= bx[2];
    if (DIM == 3) out = out || z >= bx[5] || z <= bx[4];
    if (bad) set_error(err, MPS_ERR_NAN);
    if (out) set_error(err, MPS_ERR_BOX);
}

// PREPDATA (functions.cu:2688-2746): roll state, flag ERROR#1 / ERROR#2
template <int DIM>
__global__ void k_commit(int n, Box B, const int* __restrict__ ptype,
                         const double* __restrict__ x, const double* __restrict__ y,
                         const double* __restrict__ z, double* __restrict__ u,
                         double* __restrict__ v, double* __restrict__ w, double* __restrict__ p,
                         const double* __restrict__ un, const double* __restrict__ vn,
                         const double* __restrict__ wn, const double* __restrict__ pnew,
                         unsigned int* err)
{
    int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= n) return;
    double pI = pnew[I];
    p[I] = pI;
    double uI = u[I], vI = v[I], wI = DIM == 3 ? w[I] : 0.0;
    if (ptype[I] > 0) {
        uI = un[I]; vI = vn[I];
        u[I] = uI; v[I] = vI;
        if (DIM == 3) { wI = wn[I]; w[I] = wI; }
    }
    commit_checks<DIM>(B, I, x[I], y[I], DIM == 3 ? z[I] : 0.0, uI, vI, wI, pI, err);
}

// k_collision_apply and k_commit in one launch
template <int DIM>
__global__ void k_collision_commit(int n, Box B, const int* __restrict__ ptype,
                                   double* __restrict__ x, double* __restrict__ y,
                                   double* __restrict__ z, double* __restrict__ u,
                                   double* __restrict__ v, double* __restrict__ w,
                                   double* __restrict__ p, double* __restrict__ un,
                                   double* __restrict__ vn, double* __restrict__ wn,
                                   const double* __restrict__ pnew, const double* __restrict__ xo,
                                   const double* __restrict__ yo, const double* __restrict__ zo,
                                   const double* __restrict__ uo, const double* __restrict__ vo,
                                   const double* __restrict__ wo, double4* __restrict__ P4,
                                   unsigned int* err)
{
    int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= n) return;
    const double pI = pnew[I];
    p[I] = pI;
    double xi, yi, zi = 0.0, uI, vI, wI = 0.0;
    if (ptype[I] > 0) {
        double4 pi = P4[I];
        pi.x = xi = xo[I];
        pi.y = yi = yo[I];
        uI = uo[I];
        vI = vo[I];
        x[I] = xi;
        y[I] = yi;
        un[I] = uI;
        vn[I] = vI;
        u[I] = uI;
        v[I] = vI;
        if (DIM == 3) {
            pi.z = zi = zo[I];
            wI = wo[I];
            z[I] = zi;
            wn[I] = wI;
            w[I] = wI;
        }
        P4[I] = pi;
    } else {
        xi = x[I];
        yi = y[I];
        uI = u[I];
        vI = v[I];
        if (DIM == 3) { zi = z[I]; wI = w[I]; }
    }
    commit_checks<DIM>(B, I, xi, yi, zi, uI, vI, wI, pI, err);
}

Lists lists(mps_ctx* c, int which)
{
    Lists L;
    L.cap = which == 0 ? c->cap_l : c->cap_s;
    L.nbr = which == 0 ? c->nbr_l : c->nbr_s;
    L.len = which == 0 ? c->len_l : c->len_s;
    return L;
}

Phys phys(mps_ctx* c)
{
    Phys P;
    const mps_config& f = c->cfg;
    P.rho1 = f.rho1; P.rho2 = f.rho2; P.nu1 = f.nu1; P.nu2 = f.nu2; P.n0 = c->n0_s;
    P.meu0 = f.meu0; P.n_pl = f.n_pl; P.phi = f.phi; P.cohes = f.cohes; P.cs = f.cs; P.l0 = f.l0;
    P.mind2 = sqrt_cut(f.coll / 10, false);
    P.fluid2_type = f.fluid2_type;
    P.wk = make_wk(f.ktype, f.re_s);
    return P;
}

Box box(mps_ctx* c)
{
    const mps_config& f = c->cfg;
    Box B{f.xmin, f.xmax, f.ymin, f.ymax, f.zmin, f.zmax, f.l0, f.dt, f.velcor,
          c->nscenes > 1 ? c->scene : nullptr, c->sbox};
    return B;
}

#define LAUNCH_DIM(kern, ...)                                                             \
    do {                                                                                  \
        if (c->cfg.dim == 3) kern<3><<<grid_blocks(c->n), kBlock, 0, c->stream>>>(__VA_ARGS__); \
        else kern<2><<<grid_blocks(c->n), kBlock, 0, c->stream>>>(__VA_ARGS__);           \
        vmps_count_launch(1);                                                             \
    } while (0)

inline int group_blocks(long n, int G) { return (int)((n * G + kBlock - 1) / kBlock); }

// G lanes per PND-radius row: SmallG, or twice that when the autotuner
// chose the wide form (ctx->tune_small_wide)
#define LAUNCH_SMALL_AS(KERN, ...)                                                        \
    do {                                                                                  \
        constexpr int G3 = SmallG<3>::G, G2 = SmallG<2>::G;                               \
        const bool wide = c->tune_small_wide != 0;                                        \
        if (c->cfg.dim == 3) {                                                            \
            if (wide) KERN(3, 2 * G3)<<<group_blocks(c->n, 2 * G3), kBlock, 0, c->stream>>>(__VA_ARGS__); \
            else KERN(3, G3)<<<group_blocks(c->n, G3), kBlock, 0, c->stream>>>(__VA_ARGS__); \
        } else {                                                                          \
            if (wide) KERN(2, 2 * G2)<<<group_blocks(c->n, 2 * G2), kBlock, 0, c->stream>>>(__VA_ARGS__); \
            else KERN(2, G2)<<<group_blocks(c->n, G2), kBlock, 0, c->stream>>>(__VA_ARGS__); \
        }                                                                                 \
        vmps_count_launch(1);                                                             \
    } while (0)
// a kernel over kernel-function values: its form for type 2, or for any type
#define LAUNCH_SMALL_W(kern, ...)                                                         \
    do {                                                                                  \
        if (c->cfg.ktype == 2) LAUNCH_SMALL_AS(kern##_2, __VA_ARGS__);                    \
        else LAUNCH_SMALL_AS(kern##_any, __VA_ARGS__);                                    \
    } while (0)
#define k_pnd_2(D, G) k_pnd<D, G, 2>
#define k_pnd_any(D, G) k_pnd<D, G, 0>
#define k_vfraction_2(D, G) k_vfraction<D, G, 2>
#define k_vfraction_any(D, G) k_vfraction<D, G, 0>
#define k_viscosity_2(D, G) k_viscosity<D, G, 2>
#define k_viscosity_any(D, G) k_viscosity<D, G, 0>
#define k_sps1_2(D, G) k_sps1<D, G, 2>
#define k_sps1_any(D, G) k_sps1<D, G, 0>
#define k_sps2_2(D, G) k_sps2<D, G, 2>
#define k_sps2_any(D, G) k_sps2<D, G, 0>
#define k_predict_p_2(D, G) k_predict_p<D, G, 2>
#define k_predict_p_any(D, G) k_predict_p<D, G, 0>
#define k_pressgrad_2(D, G) k_pressgrad<D, G, 2, false>
#define k_pressgrad_any(D, G) k_pressgrad<D, G, 0, false>
#define k_pressgrad_move_2(D, G) k_pressgrad<D, G, 2, true>
#define k_pressgrad_move_any(D, G) k_pressgrad<D, G, 0, true>
#define k_pnd32_2(D, G) k_pnd32<D, G, 2>
#define k_pnd32_any(D, G) k_pnd32<D, G, 0>
#define k_pressgrad32_2(D, G) k_pressgrad32<D, G, 2>
#define k_pressgrad32_any(D, G) k_pressgrad32<D, G, 0>
#define k_collision_form(D, G) k_collision<D, G>
#define LAUNCH_GROUP(G, kern, ...)                                                        \
    do {                                                                                  \
        if (c->cfg.dim == 3)                                                              \
            kern<3><<<group_blocks(c->n, G), kBlock, 0, c->stream>>>(__VA_ARGS__);        \
        else                                                                              \
            kern<2><<<group_blocks(c->n, G), kBlock, 0, c->stream>>>(__VA_ARGS__);        \
        vmps_count_launch(1);                                                             \
    } while (0)
#define LAUNCH_WARP(kern, ...)                                                            \
    do {                                                                                  \
        if (c->cfg.dim == 3)                                                              \
            kern<3><<<group_blocks(c->n, 32), kBlock, 0, c->stream>>>(__VA_ARGS__);       \
        else                                                                              \
            kern<2><<<group_blocks(c->n, 32), kBlock, 0, c->stream>>>(__VA_ARGS__);       \
        vmps_count_launch(1);                                                             \
    } while (0)

}  // namespace

// FP32 copies relative to (x0, y0, z0); w = ptype when given, else 0
__global__ void k_pack_f(int n, const double* __restrict__ x, const double* __restrict__ y,
                         const double* __restrict__ z, double x0, double y0, double z0,
                         const int* __restrict__ ptype, float4* __restrict__ P4f)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        P4f[i] = make_float4((float)(x[i] - x0), (float)(y[i] - y0), (float)(z[i] - z0),
                             ptype ? (float)ptype[i] : 0.f);
}

int vmps_pack(mps_ctx* c)
{
    const mps_config& f = c->cfg;
    k_pack_f<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->x, c->y, c->z, f.xmin, f.ymin,
                                                          f.dim == 3 ? f.zmin : 0.0, c->ptype,
                                                          c->P4f);
    vmps_count_launch(1);
    if (f.precision >= 1) {
        k_pack_f<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->u, c->v, c->w, 0.0, 0.0,
                                                              0.0, nullptr, c->U4f);
        vmps_count_launch(1);
    }
    k_pack<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->x, c->y, c->z, c->ptype, c->P4);
    k_pack<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->u, c->v, c->w, nullptr, c->U4);
    vmps_count_launch(2);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

// the packed velocities alone (mps_step_io's deferred velocities)
int vmps_pack_u(mps_ctx* c)
{
    if (c->cfg.precision >= 1) {
        k_pack_f<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->u, c->v, c->w, 0.0, 0.0,
                                                              0.0, nullptr, c->U4f);
        vmps_count_launch(1);
    }
    k_pack<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(c->n, c->u, c->v, c->w, nullptr, c->U4);
    vmps_count_launch(1);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_pnd(mps_ctx* c, int at_star, int correct, int which, double* out, bool track_max,
             bool with_bcon)
{
    const BconOut B{with_bcon ? c->bcon : nullptr, c->ptype, c->n0_s, c->cfg.dirichlet};
    double re = which == 0 ? c->cfg.re_l : c->cfg.re_s;
    // the maximum is wanted once (n0); per step its atomics would all hit
    // one address
    unsigned long long* dmax = track_max ? c->d_max : nullptr;
    const double4* P = at_star ? c->P4s : c->P4;
    WK wk = make_wk(c->cfg.ktype, re);
    if (which == 0) {
        if (c->cfg.dim == 3)
            k_pnd<3, 32, 0><<<group_blocks(c->n, 32), kBlock, 0, c->stream>>>(
                c->n, lists(c, 0), P, wk, correct, c->cfg.ncorrection, out, dmax, B);
        else
            k_pnd<2, 32, 0><<<group_blocks(c->n, 32), kBlock, 0, c->stream>>>(
                c->n, lists(c, 0), P, wk, correct, c->cfg.ncorrection, out, dmax, B);
        vmps_count_launch(1);
    } else if (at_star && !correct && c->cfg.precision == 2 && c->P4sf) {
        // precision 2: n* from the FP32 predicted positions
        LAUNCH_SMALL_W(k_pnd32, c->n, lists(c, 1), c->P4sf, make_wkf(wk), out);
    } else {
        LAUNCH_SMALL_W(k_pnd, c->n, lists(c, 1), P, wk, correct, c->cfg.ncorrection, out, dmax, B);
    }
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_bcon(mps_ctx* c)
{
    k_bcon<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(
        c->n, c->ptype, c->nds, c->n0_s, c->cfg.dirichlet, c->bcon,
        c->cfg.ppe_at_predicted ? c->P4s : nullptr);
    c->p4s_bcon = c->cfg.ppe_at_predicted != 0;
    vmps_count_launch(1);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

// The explicit stages of a step: V_FRACTION, VISCOSITY, PREDICTION, PNUMSTAR and
// (method 1) BCON, with the passes that need no neighbours in one launch and BCON
// in PNUMSTAR's pass.  The same results as the stages one by one, but for the w
// slot of the predicted positions, which BCON fills and the pressure assembly
// fills anew when it forms CG's starting residual; elsewhere BCON runs by itself.
int vmps_explicit(mps_ctx* c)
{
    const mps_config& f = c->cfg;
    const bool no_c = c->fp2 == 0, by_kind = f.fluid2_type == 0;
    k_explicit_begin<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(
        c->n, c->x, c->y, c->z, c->pnew, c->ptype, f.nu1 * f.rho1, f.nu2 * f.rho2, c->PP4,
        no_c ? c->C : nullptr, by_kind ? c->meu : nullptr);
    vmps_count_launch(1);
    int r = MPS_OK;
    if (!no_c) r = vmps_vfraction(c);
    if (r == MPS_OK && !by_kind) r = vmps_viscosity(c);
    if (r == MPS_OK) r = vmps_predict(c, true);
    if (r != MPS_OK) return r;
    const bool join = f.method != 3 && f.precision != 2 && f.ppe_at_predicted && !f.srcopt &&
                      (f.warm_start == 1 || vmps_gnn_in_use(c));
    r = vmps_pnd(c, 1, 0, 1, c->nds, false, join);
    if (r == MPS_OK && f.method != 3 && !join) r = vmps_bcon(c);
    return r;
}

int vmps_vfraction(mps_ctx* c)
{
    // without second-fluid particles every sum2 is 0, so C = 0 everywhere
    // (sum1 = 0 also gives 0): no neighbour pass
    if (c->fp2 == 0) {
        VMPS_CUDA(c, cudaMemsetAsync(c->C, 0, sizeof(double) * c->n, c->stream));
        return MPS_OK;
    }
    LAUNCH_SMALL_W(k_vfraction, c->n, lists(c, 1), c->ptype, c->P4, make_wk(c->cfg.ktype, c->cfg.re_s),
               c->cfg.fraction_method, c->C);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_viscosity(mps_ctx* c)
{
    LAUNCH_SMALL_W(k_viscosity, c->n, lists(c, 1), phys(c), c->ptype, c->P4, c->un, c->vn, c->wn, c->C,
               c->phat, c->meu);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_sps(mps_ctx* c)
{
    Phys P = phys(c);
    LAUNCH_SMALL_W(k_sps1, c->n, lists(c, 1), P, c->ptype, c->P4, c->un, c->vn, c->wn, c->S6, c->neut);
    LAUNCH_SMALL_W(k_sps2, c->n, lists(c, 1), P, c->ptype, c->P4, c->S6, c->neut, c->t1, c->t2, c->t3);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_predict(mps_ctx* c, bool packed)
{
    const mps_config& f = c->cfg;
    PredArgs A;
    A.ws = make_wk(f.ktype, f.re_s);
    A.wl = make_wk(f.ktype, f.re_l);
    A.n0_s = c->n0_s;
    // 4*DT/(lambda*n0) of the viscous term (functions.cu:2361; "4" is the
    // reference's 2*d with d = 2, kept in 3D as well)
    A.visc_coef = 4 * f.dt / (c->lambda_l * c->n0_l);
    A.dt = f.dt; A.gx = f.gx; A.gy = f.gy; A.gz = f.gz; A.relaxp = f.relaxp;
    A.rho1 = f.rho1; A.rho2 = f.rho2;
    // the same products VISCOSITY forms (k_viscosity, fluid2_type 0)
    A.meu1 = f.nu1 * f.rho1;
    A.meu2 = f.nu2 * f.rho2;
    if (!packed) {
        k_explicit_begin<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(
            c->n, c->x, c->y, c->z, c->pnew, c->ptype, 0.0, 0.0, c->PP4, nullptr, nullptr);
        vmps_count_launch(1);
    }
    LAUNCH_SMALL_W(k_predict_p, c->n, lists(c, 1), A, c->P4, c->PP4, c->phat, c->rho, c->pres_x,
                 c->pres_y, c->pres_z);
    // without SPS, neut is 0 and the eddy-viscosity sums are left out
#define PRED32(D, T, K, B)                                                                    \
    k_predict32<D, T, K, B><<<group_blocks(c->n, kPred32G), kBlock, 0, c->stream>>>(                 \
        c->n, lists(c, 0), A, make_wkf(A.wl), c->meu, c->P4, c->U4, c->P4f, c->U4f, c->pres_x, \
        c->pres_y, c->pres_z, c->neut, c->t1, c->t2, c->t3, c->xs, c->ys, c->zs, c->us, c->vs,  \
        c->ws, c->P4s, c->P4sf, make_double3(f.xmin, f.ymin, f.dim == 3 ? f.zmin : 0.0))
#define PRED64(D, T, K, B)                                                                    \
    k_predict<D, T, K, B><<<(int)(((long)c->n * kPredG + kPredThreads - 1) / kPredThreads),   \
                            kPredThreads, 0, c->stream>>>(                     \
        c->n, lists(c, 0), A, c->meu, c->P4, c->U4, c->pres_x, c->pres_y, c->pres_z, c->neut,  \
        c->t1, c->t2, c->t3, c->xs, c->ys, c->zs, c->us, c->vs, c->ws, c->P4s)
    const bool turb = f.turb != 0;
    c->p4s_bcon = false;  // P4s.w is ptype again until BCON
    const bool k2 = f.ktype == 2, by_kind = f.fluid2_type == 0;
#define PRED_B(P, D, T, K) do { if (by_kind) P(D, T, K, true); else P(D, T, K, false); } while (0)
#define PRED_K(P, D, T) do { if (k2) PRED_B(P, D, T, 2); else PRED_B(P, D, T, 0); } while (0)
#define PRED_T(P, D) do { if (turb) PRED_K(P, D, true); else PRED_K(P, D, false); } while (0)
    if (f.precision >= 1) {  // FP32 neighbour sums
        if (f.dim == 3) PRED_T(PRED32, 3);
        else PRED_T(PRED32, 2);
    } else {
        if (f.dim == 3) PRED_T(PRED64, 3);
        else PRED_T(PRED64, 2);
    }
#undef PRED_T
#undef PRED_K
#undef PRED_B
#undef PRED32
#undef PRED64
    vmps_count_launch(1);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_pressure_wc(mps_ctx* c)
{
    const mps_config& f = c->cfg;
    k_pressure_wc<<<grid_blocks(c->n), kBlock, 0, c->stream>>>(
        c->n, c->ptype, c->C, c->nds, c->n0_s, f.beta_fs, f.c01, f.c02, f.rho1, f.rho2, f.pmin,
        f.pmax, c->pnew);
    vmps_count_launch(1);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_phat(mps_ctx* c)
{
    const int G = (c->cfg.dim == 3 ? SmallG<3>::G : SmallG<2>::G) * (c->tune_small_wide ? 2 : 1);
    if (G == 16)
        k_phat<16><<<group_blocks(c->n, 16), kBlock, 0, c->stream>>>(c->n, lists(c, 1), c->pnew,
                                                                     c->phat, c->PH, c->PH32);
    else if (G == 8)
        k_phat<8><<<group_blocks(c->n, 8), kBlock, 0, c->stream>>>(c->n, lists(c, 1), c->pnew,
                                                                   c->phat, c->PH, c->PH32);
    else
        k_phat<4><<<group_blocks(c->n, 4), kBlock, 0, c->stream>>>(c->n, lists(c, 1), c->pnew,
                                                                   c->phat, c->PH, c->PH32);
    vmps_count_launch(1);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

// Up to this many particles a step's EULERINTEGRATION runs in PRESSGRAD's pass: it
// saves a launch (3 us of a 180 us step), but one lane in four moves a particle
// there (476 k particles: 169 us against 101 + 28 us)
constexpr int kMoveMax = 65536;

int vmps_pressgrad(mps_ctx* c, bool move)
{
    const mps_config& f = c->cfg;
    GradArgs A;
    A.wk = make_wk(f.ktype, f.re_s);
    A.coef = f.relaxp * (2.0 * f.dt / c->n0_s);
    A.vmax = f.vmax;
    A.kh = f.kh;
    if (f.precision == 2)
        LAUNCH_SMALL_W(k_pressgrad32, c->n, lists(c, 1), A, make_wkf(A.wk), c->ptype, c->PH32,
                     c->P4sf, c->rho, c->us, c->vs, c->ws, c->un, c->vn, c->wn);
    else if (move && c->n <= kMoveMax)
        LAUNCH_SMALL_W(k_pressgrad_move, c->n, lists(c, 1), A, c->ptype, c->PH, c->P4s, c->rho,
                       c->us, c->vs, c->ws, c->un, c->vn, c->wn,
                       MoveArgs{box(c), c->x, c->y, c->z, c->P4});
    else
        LAUNCH_SMALL_W(k_pressgrad, c->n, lists(c, 1), A, c->ptype, c->PH, c->P4s, c->rho, c->us,
                       c->vs, c->ws, c->un, c->vn, c->wn, MoveArgs{});
    VMPS_CUDA(c, cudaGetLastError());
    if (move && (f.precision == 2 || c->n > kMoveMax)) return vmps_integrate(c);
    return MPS_OK;
}

int vmps_integrate(mps_ctx* c)
{
    LAUNCH_DIM(k_integrate, c->n, box(c), c->ptype, c->x, c->y, c->z, c->un, c->vn, c->wn, c->P4);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

static void collide(mps_ctx* c)
{
    const mps_config& f = c->cfg;
    CollArgs A{sqrt_cut(f.coll, true), f.cc, f.dt, f.rho1, f.rho2};
    // new states to the *c scratch arrays, then copied over in place
    LAUNCH_SMALL_AS(k_collision_form, c->n, lists(c, 1), A, c->ptype, c->oid, c->P4, c->un, c->vn,
                    c->wn, c->xc, c->yc, c->zc, c->uc, c->vc, c->wc);
}

int vmps_collision(mps_ctx* c)
{
    collide(c);
    LAUNCH_DIM(k_collision_apply, c->n, c->ptype, c->x, c->y, c->z, c->un, c->vn, c->wn, c->xc,
               c->yc, c->zc, c->uc, c->vc, c->wc, c->P4);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

// COLLISION2 and PREPDATA of a step
int vmps_collision_commit(mps_ctx* c)
{
    collide(c);
    LAUNCH_DIM(k_collision_commit, c->n, box(c), c->ptype, c->x, c->y, c->z, c->u, c->v, c->w, c->p,
               c->un, c->vn, c->wn, c->pnew, c->xc, c->yc, c->zc, c->uc, c->vc, c->wc, c->P4,
               c->d_err);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}

int vmps_commit(mps_ctx* c)
{
    LAUNCH_DIM(k_commit, c->n, box(c), c->ptype, c->x, c->y, c->z, c->u, c->v, c->w, c->p, c->un,
               c->vn, c->wn, c->pnew, c->d_err);
    VMPS_CUDA(c, cudaGetLastError());
    return MPS_OK;
}
