// FP64 tangent of linear cells through element matrices: SimpleAssembler::BuildMatrix
// (nuto/mechanics/cell/SimpleAssembler.cpp:100-156) of MomentumBalance::Hessian0 with LinearElastic
// (nuto/mechanics/integrands/MomentumBalance.h:36-46) and GradientDamage::Hessian0
// (nuto/mechanics/integrands/GradientDamage.h:92-120) for Quad4 and Hex8 cells with the two-point rule. k_cell_matrices64
// integrates every cell's element matrix once, k_rows_from_slabs (rows.cuh) adds them into the CSR rows: no atomics, the
// values are bitwise reproducible.
//
// Bound by the FP64 pipe (2 lanes per clock and SM); what is saved against an element kernel that integrates each ordered
// node pair on its own:
// - the material tangent is lambda m m^T + mu diag(2..2, 1..1) with one ratio rho = lambda / mu for all points (LinearElastic;
//   LinearElasticDamage with FULL damage application), so a displacement block is rho S + S^T + tr(S) I with the one sum
//   S = sum over the points of mu w g_a g_b^T, and the block of (b, a) is the transpose: 9 multiply-adds per point and
//   unordered pair instead of 33 per ordered pair;
// - the coupling blocks sum_q P_a(q) N_b(q) are transposed interpolations, sum-factorised over the points (24 multiply-adds
//   per row of 8 blocks instead of 64, sumfac.cuh).
// 8,800 FP64 instructions per Hex8 gradient-damage cell against about 33,000; 64^3 14.46 -> 4.66 ms, 40^3 3.57 -> 1.18 ms,
// 17^3 317 -> 118 us, 200^2 Quad4 elastic 109 -> 39 us (k_cell_matrices64 at 90 % of the FP64 pipe; the gather of 8 KB
// per cell 12 % of the time). The same values serve NUTO_GPU_FP64X, whose double-float products took 2.03 ms at 40^3.
#include "rows.cuh"
#include "sumfac.cuh"

#include <algorithm>
#include <cfloat>

namespace nuto_gpu
{

namespace
{

template <int DIM, bool GD>
struct Cell64
{
    static constexpr int nd = SumFac<DIM>::nd, nip = nd;
    static constexpr int vd = DIM == 2 ? 3 : 6;
    static constexpr int nf = DIM + (GD ? 1 : 0);
    static constexpr int threads = 64;
    static constexpr int cpb = threads / nip; // one thread per (cell, point) and per (cell, node)
    static constexpr int pairs = nd * (nd + 1) / 2;
    // per point: the node gradients, the same times mu w; gradient damage: the Voigt vectors of the coupling blocks, the
    // eeq-gradient coupling vector, w and c g w (all but the gradients scaled as their use below wants them)
    static constexpr int oG = 0, oM = nd * DIM, oS = 2 * nd * DIM, oT = oS + vd, oC = oT + vd, oW = oC + DIM;
    static constexpr int rec = GD ? oW + 2 : oS;
    static constexpr int ng = SumFac<DIM>::ng;
};

// node pair p of the upper triangle (a <= b), row by row
template <int ND>
__device__ __forceinline__ void UnorderedPair(int p, int& a, int& b)
{
    a = 0;
    int row = ND;
    while (p >= row)
    {
        p -= row;
        --row;
        ++a;
    }
    b = a + p;
}

template <int DIM, bool GD>
__global__ void __launch_bounds__(Cell64<DIM, GD>::threads) k_cell_matrices64(CellArgs a, LawParams L,
                                                                              const double* __restrict__ u,
                                                                              double* __restrict__ em)
{
    using C = Cell64<DIM, GD>;
    using S = SumFac<DIM>;
    using SL = Slab<DIM, C::nd, GD>;
    constexpr int ND = C::nd, NIP = C::nip, VD = C::vd, CPB = C::cpb, REC = C::rec;
    extern __shared__ double sm64[];
    double* sRec = sm64;                        // [NIP][REC][CPB]
    double* sGrad = sRec + NIP * REC * CPB;     // [NF][ng][CPB], later the (eeq, eeq) sums [ND][ND][CPB]
    double* sEn = sGrad + (C::nf * C::ng > ND * ND ? C::nf * C::ng : ND * ND) * CPB; // nodal eeq [ND][CPB]
    const int64_t n = a.nCells;
    const int64_t cell0 = static_cast<int64_t>(blockIdx.x) * CPB;
    auto at = [&](int q, int k, int cl) -> double& { return sRec[(q * REC + k) * CPB + cl]; };

    // natural gradients of the displacement components and of eeq
    for (int it = threadIdx.x; it < CPB * C::nf; it += C::threads)
    {
        const int cl = it % CPB, fl = it / CPB;
        const int64_t e = cell0 + cl;
        if (e >= n)
            continue;
        const bool eq = GD && fl == DIM;
        const int32_t* conn = eq ? a.connE : a.connD;
        const int64_t* gdof = eq ? a.gdofE : a.gdofD;
        const int comp = eq ? 0 : fl;
        double v[ND], g[S::ng];
#pragma unroll
        for (int nd = 0; nd < ND; ++nd)
        {
            const int64_t gd = gdof[NG_IDX(conn[static_cast<int64_t>(nd) * n + e], eq ? a.nNodesE : a.nNodesD, 2)];
            v[nd] = u[NG_IDX(gd + comp, a.nDofs, 3)];
            if (eq)
                sEn[nd * CPB + cl] = v[nd];
        }
        SfForward<double, DIM, false>(v, g, nullptr);
#pragma unroll
        for (int k = 0; k < S::ng; ++k)
            sGrad[(fl * S::ng + k) * CPB + cl] = g[k];
    }
    __syncthreads();

    // the law and the node gradients of every point
    {
        const int cl = threadIdx.x % CPB, q = threadIdx.x / CPB;
        const int64_t e = cell0 + cl;
        if (e < n)
        {
            const double* Jq = a.jac + NG_IDX(static_cast<int64_t>(q) * (1 + DIM * DIM) * n + e, a.jacSize, 6);
            const double wdj = Jq[0];
            // per-cell Young's modulus factor: scales the material tangent and dsigma/domega (displacement rows)
            const double wdjE = a.escale ? wdj * a.escale[e] : wdj;
            double muw;
            if (!GD)
                muw = L.C33 * wdjE;
            else
            {
                double J[DIM][DIM], G[DIM][DIM], eps[VD];
#pragma unroll
                for (int j = 0; j < DIM; ++j)
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                        J[j][d] = Jq[(1 + j * DIM + d) * n];
#pragma unroll
                for (int c = 0; c < DIM; ++c)
#pragma unroll
                    for (int j = 0; j < DIM; ++j)
                        G[c][j] = sGrad[(c * S::ng + SfGradIndex<DIM>(j, q)) * CPB + cl];
                StrainFromNatural<double, DIM>(G, J, eps);
                // eeq in the order of the history update and of the other tangents: a converged loading point has
                // eeq = kappa there, and the loading test must find it loading
                double eeq = 0.;
#pragma unroll
                for (int nd = 0; nd < ND; ++nd)
                    eeq = fma(a.tabN_D[q * ND + nd], sEn[nd * CPB + cl], eeq);
                const double kh = a.kappa[NG_IDX(e * NIP + q, n * NIP, 7)];
                const double kap = kh > eeq ? kh : eeq;
                const bool loading = eeq >= kh;
                double phi = 1., dom = 0.;
                if (!(kap < L.kappa0))
                {
                    const double ki = 1. / kap, ex = L.alpha * exp(L.beta * (L.kappa0 - kap));
                    const double k0i = L.kappa0 * ki;
                    phi = 1. - (1. - k0i * ((1. - L.alpha) + ex)); // as DamageIntegrity
                    dom = k0i * ((ki + L.beta) * ex + (1. - L.alpha) * ki);
                }
                if (!loading)
                    dom = 0.;
                double g = 1., dgdw = 0.;
                if (L.interaction != NUTO_GPU_INTERACTION_CONSTANT)
                {
                    g = InteractionFactor<double>(L, 1. - phi);
                    dgdw = InteractionDerivative<double>(L, 1. - phi);
                }
                muw = phi * L.muD * wdjE;
                // (disp, eeq): B^T (dsigma/domega omega' kappa') N with dsigma/domega = -(lambda tr + 2 mu eps); the
                // factor of the sum-factorised transpose goes in here
                double tr = eps[0] + eps[1];
                if (DIM == 3)
                    tr += eps[2];
                const double f = -S::valScale * dom * wdjE, t = L.lamD * tr, fm = f * L.muD;
#pragma unroll
                for (int v = 0; v < VD; ++v)
                    at(q, C::oS + v, cl) = v < DIM ? f * (L.m2G * eps[v] + t) : fm * eps[v];
                // (eeq, disp): -N^T (deps_eq/deps)^T B
                double dn[VD];
                MisesDerivative<double, DIM>(L, eps, dn);
                const double fn = -S::valScale * wdj;
#pragma unroll
                for (int v = 0; v < VD; ++v)
                    at(q, C::oT + v, cl) = fn * dn[v];
                // (eeq, eeq): (w N_a + gs_a) N_b + c g w (g_a . g_b), gs_a = c g' omega' kappa' w (grad eeq . g_a)
                const double sc = S::valScale * L.c * dgdw * dom * wdj;
                double ge[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    ge[d] = 0.;
                if (sc != 0.)
                {
#pragma unroll
                    for (int j = 0; j < DIM; ++j)
#pragma unroll
                        for (int d = 0; d < DIM; ++d)
                            ge[d] += sGrad[(DIM * S::ng + SfGradIndex<DIM>(j, q)) * CPB + cl] * J[j][d];
                }
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    at(q, C::oC + d, cl) = sc * ge[d];
                at(q, C::oW, cl) = S::valScale * wdj;
                at(q, C::oW + 1, cl) = L.c * g * wdj;
            }
            const double* Gq = a.geo64 + NG_IDX(static_cast<int64_t>(q) * a.geoStride * n + e, a.geoSize, 6);
#pragma unroll
            for (int k = 0; k < ND * DIM; ++k)
            {
                const double g = Gq[(1 + k) * n];
                at(q, C::oG + k, cl) = g;
                at(q, C::oM + k, cl) = muw * g;
            }
        }
    }
    __syncthreads();

    // displacement blocks of the unordered pairs and the gradient part of the (eeq, eeq) entries
    const double mu0 = GD ? L.muD : L.C33;
    const double rho = mu0 != 0. ? (GD ? L.lamD : L.C12) / mu0 : 0.;
    for (int it = threadIdx.x; it < CPB * C::pairs; it += C::threads)
    {
        const int cl = it % CPB;
        int ia, ib;
        UnorderedPair<ND>(it / CPB, ia, ib);
        const int64_t e = cell0 + cl;
        if (e >= n)
            continue;
        double s[DIM][DIM], dd = 0.;
#pragma unroll
        for (int k = 0; k < DIM; ++k)
#pragma unroll
            for (int l = 0; l < DIM; ++l)
                s[k][l] = 0.;
#pragma unroll 2
        for (int q = 0; q < NIP; ++q)
        {
            double m[DIM], gb[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
            {
                m[d] = at(q, C::oM + ia * DIM + d, cl);
                gb[d] = at(q, C::oG + ib * DIM + d, cl);
            }
#pragma unroll
            for (int k = 0; k < DIM; ++k)
#pragma unroll
                for (int l = 0; l < DIM; ++l)
                    s[k][l] += m[k] * gb[l];
            if (GD)
            {
                double gab = at(q, C::oG + ia * DIM, cl) * gb[0];
#pragma unroll
                for (int d = 1; d < DIM; ++d)
                    gab += at(q, C::oG + ia * DIM + d, cl) * gb[d];
                dd += at(q, C::oW + 1, cl) * gab;
            }
        }
        double tr = s[0][0];
#pragma unroll
        for (int k = 1; k < DIM; ++k)
            tr += s[k][k];
        double* rowA = em + (NG_IDX(e, n, 84) * ND + ia) * SL::size + ib * DIM;
        double* rowB = em + (e * ND + ib) * SL::size + ia * DIM;
#pragma unroll
        for (int k = 0; k < DIM; ++k)
#pragma unroll
            for (int l = 0; l < DIM; ++l)
            {
                const double v = rho * s[k][l] + (k == l ? s[l][k] + tr : s[l][k]);
                rowA[k * SL::nc + l] = v;
                if (ia != ib)
                    rowB[l * SL::nc + k] = v;
            }
        if (GD)
        {
            sGrad[(ia * ND + ib) * CPB + cl] = dd;
            sGrad[(ib * ND + ia) * CPB + cl] = dd;
        }
    }
    if constexpr (GD)
    {
        __syncthreads();
        // coupling blocks: thread (cell, a) the (disp a, eeq) and (eeq a, eeq) rows over all b, then (eeq, disp a)
        const int cl = threadIdx.x % CPB, ia = threadIdx.x / CPB;
        const int64_t e = cell0 + cl;
        if (e >= n)
            return;
        double f[DIM + 1][NIP], o[ND];
#pragma unroll
        for (int q = 0; q < NIP; ++q)
        {
            double g[DIM], sv[VD], P[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                g[d] = at(q, C::oG + ia * DIM + d, cl);
#pragma unroll
            for (int v = 0; v < VD; ++v)
                sv[v] = at(q, C::oS + v, cl);
            BtS<double, DIM>(g, sv, P);
            double z = at(q, C::oW, cl) * a.tabN_D[q * ND + ia];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
            {
                f[d][q] = P[d];
                z += at(q, C::oC + d, cl) * g[d];
            }
            f[DIM][q] = z;
        }
        double* slab = em + (e * ND + ia) * SL::size;
#pragma unroll
        for (int k = 0; k <= DIM; ++k)
        {
            SfValuesToNodes<double, DIM>(f[k], o);
            double* row = slab + k * SL::nc + ND * DIM;
#pragma unroll
            for (int b = 0; b < ND; ++b)
                row[b] = k < DIM ? o[b] : o[b] + sGrad[(ia * ND + b) * CPB + cl];
        }
#pragma unroll
        for (int q = 0; q < NIP; ++q)
        {
            double g[DIM], tv[VD], Q[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                g[d] = at(q, C::oG + ia * DIM + d, cl);
#pragma unroll
            for (int v = 0; v < VD; ++v)
                tv[v] = at(q, C::oT + v, cl);
            BtS<double, DIM>(g, tv, Q);
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                f[d][q] = Q[d];
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d)
        {
            SfValuesToNodes<double, DIM>(f[d], o);
#pragma unroll
            for (int r = 0; r < ND; ++r) // (eeq r, disp (ia, d))
                em[(e * ND + r) * SL::size + DIM * SL::nc + ia * DIM + d] = o[r];
        }
    }
}

// ---- Hex20 displacement cells, 3 x 3 x 3 points, LinearElastic or LocalIsotropicDamage with FULL damage -------------------
// One block per cell: (A) threads (point, component) the displacement gradient, then thread (point) the law; (B) the node
// gradients times mu w and, for the points whose rank-1 part does not vanish, P = B^T (dsigma/domega omega') w and
// Q = B^T deps_eq/deps (LocalIsotropicDamage::Tangent, nuto/mechanics/constitutive/LocalIsotropicDamage.h:59-68, 115-122);
// (C) thread = unordered node pair: rho S + S^T + tr(S) I over all points as above, and the rank-1 sums P_a Q_b^T and
// P_b Q_a^T over the loading points only. Undamaged, unloading points have P or Q = 0 exactly: their terms are left out (a
// NaN is no zero). Bound by the FP64 pipe (95 % busy): 4,525 FP64 warp instructions per cell with half of the points
// loading. 13^3: 2261 -> 607 us (the element kernel formed each ordered pair with its own lambda and mu sums and added with
// atomics), of which the gather 38 us.
constexpr int kH20Nd = 20, kH20Nip = 27, kH20Pairs = kH20Nd * (kH20Nd + 1) / 2, kH20Threads = 224;

template <bool LD>
struct H20Shared
{
    double u[kH20Nd * 3];
    double H[kH20Nip][9];
    double g[kH20Nip][kH20Nd * 3];  // node gradients
    double m[kH20Nip][kH20Nd * 3];  // the same times mu w
    double muw[kH20Nip];
    double st[LD ? kH20Nip : 1][12]; // Voigt vectors of P and Q
    double P[LD ? kH20Nip : 1][kH20Nd * 3], Q[LD ? kH20Nip : 1][kH20Nd * 3]; // compacted: loading points first
    int list[kH20Nip];
    int loading;
};

template <int KIND>
__global__ void __launch_bounds__(kH20Threads) k_cell_matrices64_h20(CellArgs a, LawParams L, const double* __restrict__ u,
                                                                     double* __restrict__ em)
{
    constexpr bool LD = KIND == NUTO_GPU_MB_LOCAL_DAMAGE;
    constexpr int ND = kH20Nd, NIP = kH20Nip;
    extern __shared__ __align__(16) unsigned char smRaw[];
    H20Shared<LD>& sh = *reinterpret_cast<H20Shared<LD>*>(smRaw);
    const int64_t n = a.nCells, e = blockIdx.x;
    const int tid = threadIdx.x;
    if (tid < ND)
    {
        const int64_t gd = a.gdofD[NG_IDX(a.connD[static_cast<int64_t>(tid) * n + e], a.nNodesD, 2)];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            sh.u[tid * 3 + c] = u[NG_IDX(gd + c, a.nDofs, 3)];
    }
    for (int it = tid; it < NIP * ND * 3; it += kH20Threads)
    {
        const int q = it / (ND * 3), k = it % (ND * 3);
        sh.g[q][k] = a.geo64[NG_IDX((static_cast<int64_t>(q) * a.geoStride + 1 + k) * n + e, a.geoSize, 6)];
    }
    __syncthreads();
    if (LD)
    {
        // in the node order of the history update (EvolutionImplicit): the loading test compares with what it stored
        for (int it = tid; it < NIP * 3; it += kH20Threads)
        {
            const int q = it % NIP, c = it / NIP;
            double h[3] = {0., 0., 0.};
#pragma unroll 5
            for (int nd = 0; nd < ND; ++nd)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    h[d] = fma(sh.u[nd * 3 + c], sh.g[q][nd * 3 + d], h[d]);
#pragma unroll
            for (int d = 0; d < 3; ++d)
                sh.H[q][c * 3 + d] = h[d];
        }
        __syncthreads();
    }
    if (tid < 32)
    {
        const int q = tid;
        bool on = false;
        if (q < NIP)
        {
            const double wdj = a.geo64[NG_IDX(static_cast<int64_t>(q) * a.geoStride * n + e, a.geoSize, 6)];
            const double wdjE = a.escale ? wdj * a.escale[e] : wdj;
            if (!LD)
                sh.muw[q] = L.C33 * wdjE;
            else
            {
                double H[3][3], eps[6];
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        H[c][d] = sh.H[q][c * 3 + d];
                StrainFromH<double, 3>(H, eps);
                const double kh = a.kappa[NG_IDX(e * NIP + q, n * NIP, 7)];
                const double eqs = MisesValue<double, 3>(L, eps);
                const double kap = eqs > kh ? eqs : kh;
                double phi = 1., dom = 0.;
                if (!(kap < L.kappa0))
                {
                    const double ki = 1. / kap, ex = L.alpha * exp(L.beta * (L.kappa0 - kap));
                    const double k0i = L.kappa0 * ki;
                    phi = 1. - (1. - k0i * ((1. - L.alpha) + ex)); // as DamageIntegrity
                    dom = k0i * ((ki + L.beta) * ex + (1. - L.alpha) * ki);
                }
                sh.muw[q] = phi * L.muD * wdjE;
                // at a converged state kappa_h is eqs itself, from the history update's own evaluation of the Mises norm, whose
                // last bits may differ: within 4 ulps below it a point is loading
                if (!(eqs >= kh - 4.0 * DBL_EPSILON * kh))
                    dom = eqs == eqs && kh == kh ? 0. : dom;
                const double tr = eps[0] + eps[1] + eps[2];
                const double f = -dom * wdjE, t = L.lamD * tr, fm = f * L.muD;
                double dk[6];
                on = !(dom == 0.) || !(eqs == eqs);
                if (on)
                {
                    MisesDerivative<double, 3>(L, eps, dk);
#pragma unroll
                    for (int v = 0; v < 6; ++v)
                    {
                        sh.st[q][v] = v < 3 ? f * (L.m2G * eps[v] + t) : fm * eps[v];
                        sh.st[q][6 + v] = dk[v];
                    }
                }
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, on);
        if (on)
            sh.list[__popc(mask & ((1u << tid) - 1u))] = q;
        if (tid == 0)
            sh.loading = __popc(mask);
    }
    __syncthreads();
    const int loading = LD ? sh.loading : 0;
    for (int it = tid; it < NIP * ND * 3; it += kH20Threads)
    {
        const int q = it / (ND * 3), k = it % (ND * 3);
        sh.m[q][k] = sh.muw[q] * sh.g[q][k];
    }
    if (LD)
    {
        for (int it = tid; it < loading * ND; it += kH20Threads)
        {
            const int j = it / ND, nd = it % ND, q = sh.list[j];
            const double g[3] = {sh.g[q][nd * 3], sh.g[q][nd * 3 + 1], sh.g[q][nd * 3 + 2]};
            BtS<double, 3>(g, sh.st[q], &sh.P[j][nd * 3]);
            BtS<double, 3>(g, sh.st[q] + 6, &sh.Q[j][nd * 3]);
        }
    }
    __syncthreads();
    if (tid >= kH20Pairs)
        return;
    int ia, ib;
    UnorderedPair<ND>(tid, ia, ib);
    double s[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l)
            s[k][l] = 0.;
#pragma unroll 3
    for (int q = 0; q < NIP; ++q)
    {
        const double* m = &sh.m[q][ia * 3];
        const double* g = &sh.g[q][ib * 3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l)
                s[k][l] += m[k] * g[l];
    }
    const double mu0 = LD ? L.muD : L.C33;
    const double rho = mu0 != 0. ? (LD ? L.lamD : L.C12) / mu0 : 0.;
    const double tr = s[0][0] + s[1][1] + s[2][2];
    double ab[3][3], ba[3][3]; // the blocks (a, b) and (b, a)
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l)
            ab[k][l] = ba[l][k] = rho * s[k][l] + (k == l ? s[l][k] + tr : s[l][k]);
    if (LD)
    {
#pragma unroll 2
        for (int j = 0; j < loading; ++j)
        {
            const double *pa = &sh.P[j][ia * 3], *pb = &sh.P[j][ib * 3], *qa = &sh.Q[j][ia * 3], *qb = &sh.Q[j][ib * 3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l)
                {
                    ab[k][l] += pa[k] * qb[l];
                    ba[k][l] += pb[k] * qa[l];
                }
        }
    }
    double* rowA = em + (NG_IDX(e, n, 84) * ND + ia) * (9 * ND) + ib * 3;
    double* rowB = em + (e * ND + ib) * (9 * ND) + ia * 3;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l)
        {
            rowA[k * 3 * ND + l] = ab[k][l];
            if (ia != ib)
                rowB[k * 3 * ND + l] = ba[k][l];
        }
}

} // namespace

bool LaunchTangent64H20(Ctx& c, const double* u, double* vals)
{
    const bool ld = c.prm.kind == NUTO_GPU_MB_LOCAL_DAMAGE;
    const CellArgs a = CellArgsOf(c);
    double* em = ElemMatsOrNull<double>(c, static_cast<size_t>(c.nCells) * kH20Nd * 9 * kH20Nd);
    if (!em)
        return false;
    const RowPlanArgs P = EnsureRowPlan(c);
    auto run = [&](auto kern, size_t smem) {
        NG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        kern<<<static_cast<unsigned>(c.nCells), kH20Threads, smem, c.stream>>>(a, c.law, u, em);
    };
    if (ld)
        run(k_cell_matrices64_h20<NUTO_GPU_MB_LOCAL_DAMAGE>, sizeof(H20Shared<true>));
    else
        run(k_cell_matrices64_h20<NUTO_GPU_MB_LINEAR_ELASTIC>, sizeof(H20Shared<false>));
    AfterLaunch(c, "k_cell_matrices64_h20");
    c.stats.kernel_launches += 1;
    LaunchWideRows<double, kH20Nd>(c, P, c.slots[c.prm.disp_slot].nNodes, em, vals);
    return true;
}

bool LaunchTangent64(Ctx& c, const double* u, double* vals)
{
    const bool gd = c.prm.kind == NUTO_GPU_GRADIENT_DAMAGE;
    const CellArgs a = CellArgsOf(c);
    const Slot& D = c.slots[c.prm.disp_slot];
    auto run = [&](auto dim, auto dmg) -> bool {
        constexpr int DIM = decltype(dim)::value;
        constexpr bool GD = decltype(dmg)::value;
        using C = Cell64<DIM, GD>;
        using SL = Slab<DIM, C::nd, GD>;
        double* em = ElemMatsOrNull<double>(c, static_cast<size_t>(c.nCells) * C::nd * SL::size);
        if (!em)
            return false;
        const RowPlanArgs P = EnsureRowPlan(c);
        if (c.slots.size() > static_cast<size_t>(GD ? 2 : 1)) // rows of slots that the integrand does not touch
            NG_CUDA(cudaMemsetAsync(vals, 0, c.nnz * sizeof(double), c.stream));
        constexpr int grad = std::max(C::nf * C::ng, C::nd * C::nd);
        constexpr size_t smem = static_cast<size_t>(C::nip * C::rec + grad + C::nd) * C::cpb * sizeof(double);
        auto kern = k_cell_matrices64<DIM, GD>;
        if (smem > 48 * 1024)
            NG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        NG_CUDA(LaunchEx(false, c.carveout, kern, dim3(static_cast<unsigned>((c.nCells + C::cpb - 1) / C::cpb)),
                         dim3(C::threads), smem, c.stream, a, c.law, u, em));
        AfterLaunch(c, "k_cell_matrices64");
        c.stats.kernel_launches += 1;
        LaunchRows<double, DIM, C::nd, GD, 4>(c, P, 0, D.nNodes, em, vals);
        return true;
    };
    using std::integral_constant;
    if (c.dim == 2)
        return gd ? run(integral_constant<int, 2>{}, integral_constant<bool, true>{})
                  : run(integral_constant<int, 2>{}, integral_constant<bool, false>{});
    return gd ? run(integral_constant<int, 3>{}, integral_constant<bool, true>{})
              : run(integral_constant<int, 3>{}, integral_constant<bool, false>{});
}

// ---- plan of the row gather, once per mesh -----------------------------------------------------------------------
namespace
{

struct PlanArgs
{
    int64_t nNodes, nCells, nEntries;
    const int64_t* gdofD;
    const int64_t* gdofE; // nullptr: no eeq rows
    const int32_t* eOf;
    const int64_t* cellPtr;
    const int32_t* cellIdx;
    const uint8_t* cellLoc;
    const int64_t* rowPtr;
    const uint8_t *rankU, *rankE;
    const int32_t *blkU, *blkE;
};

// thread it: the record of displacement node it, and slab and ranks of (entry, b) = (it / ND, it % ND) of the cell lists
template <int ND>
__global__ void __launch_bounds__(256) k_row_plan(PlanArgs A, RowPlan* __restrict__ plan, uint32_t* __restrict__ slab,
                                                  uint32_t* __restrict__ packed)
{
    const int64_t it = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (it < A.nNodes)
    {
        RowPlan p{};
        const int64_t g = A.gdofD[it];
        p.rowU = A.rowPtr[g];
        p.len = static_cast<int32_t>(A.rowPtr[g + 1] - p.rowU); // the rows of a node's components have one length
        p.first = A.cellPtr[it];
        p.cells = static_cast<int32_t>(A.cellPtr[it + 1] - p.first);
        p.bU = A.blkU[it];
        if (A.gdofE)
        {
            p.rowE = A.rowPtr[A.gdofE[A.eOf[it]]];
            p.bE = A.blkE[it];
        }
        plan[it] = p;
    }
    if (it >= A.nEntries * ND)
        return;
    const int64_t kc = it / ND;
    const int b = static_cast<int>(it % ND);
    const int64_t e = A.cellIdx[kc];
    const int ia = A.cellLoc[kc];
    if (b == 0)
        slab[kc] = static_cast<uint32_t>(e * ND + ia);
    const int64_t ridx = static_cast<int64_t>(ia * ND + b) * A.nCells + e;
    packed[it] = A.rankU[ridx] | static_cast<uint32_t>(A.rankE[ridx]) << 8;
}

} // namespace

// the plan depends on the integrand's slots: whether there are eeq rows, and which slot they are in
static int RowPlanKey(const Ctx& c)
{
    return 1 + c.prm.disp_slot + kMaxSlots * (c.prm.kind == NUTO_GPU_GRADIENT_DAMAGE ? 1 + c.prm.eeq_slot : 0);
}

bool RowPlanReady(const Ctx& c)
{
    return c.rowPlanKey == RowPlanKey(c);
}

// nodes' records, slab numbers, packed ranks
static size_t RowPlanBytes(const Ctx& c)
{
    const Slot& D = c.slots[c.prm.disp_slot];
    return static_cast<size_t>(D.nNodes) * sizeof(RowPlan) + static_cast<size_t>(c.nCells) * D.nen * (1 + D.nen) * sizeof(uint32_t);
}

RowPlanArgs EnsureRowPlan(Ctx& c)
{
    const Slot& D = c.slots[c.prm.disp_slot];
    const int64_t entries = c.nCells * D.nen;
    if (!RowPlanReady(c))
    {
        c.cellChunkEnd.clear();
        if (!c.rowPlanRoom)
        {
            c.dRowPlan.alloc(RowPlanBytes(c));
            c.rowPlanRoom = c.dRowPlan.p;
        }
        c.rowPlan = reinterpret_cast<RowPlan*>(c.rowPlanRoom);
        c.rowPlanRoom = nullptr;
        c.rowSlab = reinterpret_cast<uint32_t*>(c.rowPlan + D.nNodes);
        c.packedRanks = c.rowSlab + entries;
        const bool gd = c.prm.kind == NUTO_GPU_GRADIENT_DAMAGE;
        const int ns = static_cast<int>(c.slots.size()), dS = c.prm.disp_slot, eS = gd ? c.prm.eeq_slot : dS;
        PlanArgs A{};
        A.nNodes = D.nNodes;
        A.nCells = c.nCells;
        A.nEntries = entries;
        A.gdofD = D.dGdof.p;
        A.gdofE = gd ? c.slots[eS].dGdof.p : nullptr;
        A.eOf = gd ? c.dEOf.p : nullptr;
        A.cellPtr = D.dCellPtr.p;
        A.cellIdx = D.dCellIdx.p;
        A.cellLoc = D.dCellLoc.p;
        A.rowPtr = c.dRowPtr.p;
        A.rankU = c.pairs[dS * ns + dS].rank;
        A.rankE = c.pairs[dS * ns + eS].rank;
        A.blkU = c.pairs[dS * ns + dS].dBlk.p;
        A.blkE = c.pairs[dS * ns + eS].dBlk.p;
        const int64_t items = std::max(D.nNodes, entries * D.nen);
        auto kern = D.nen == 4 ? k_row_plan<4> : (D.nen == 20 ? k_row_plan<20> : k_row_plan<8>);
        kern<<<static_cast<unsigned>((items + 255) / 256), 256, 0, c.stream>>>(A, c.rowPlan, c.rowSlab, c.packedRanks);
        AfterLaunch(c, "k_row_plan");
        c.rowPlanKey = RowPlanKey(c);
    }
    RowPlanArgs P{};
    P.plan = c.rowPlan;
    P.slab = c.rowSlab;
    P.packed = c.packedRanks;
    P.nEntries = entries;
    P.nnz = c.nnz;
    return P;
}

template <typename T>
T* ElemMatsOrNull(Ctx& c, size_t count)
{
    ElemMats<T>* E;
    if constexpr (sizeof(T) == 4)
        E = &c.elemMats32;
    else
        E = &c.elemMats64;
    if (E->buf.n >= count)
        return E->buf.p;
    if (E->refused != 0 && count >= E->refused)
        return nullptr;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    NG_CUDA(cudaStreamIsCapturing(c.stream, &cs));
    if (cs != cudaStreamCaptureStatusNone)
        return nullptr;
    // One allocation (20 to 80 us each) with the plan where that is still to be made; the plan keeps its place as long as the
    // buffer: only a change of the pattern or of the integrand's slots, after which it is made anew, lets the buffer grow.
    const size_t plan = RowPlanReady(c) ? 0 : RowPlanBytes(c), matrices = (count * sizeof(T) + 255) / 256 * 256;
    const size_t bytes = matrices + plan;
    bool room = true;
    // The element kernel needs no scratch, so a large FP64 problem may have just the memory for its solver. Asking for the free
    // memory costs as much as a small assembly: below this size (1 GB of tangent at most) the attempt alone decides.
    if (sizeof(T) == 8 && bytes >= (size_t(256) << 20))
    {
        size_t free = 0, total = 0;
        NG_CUDA(cudaMemGetInfo(&free, &total));
        room = bytes + SolverBytesToCome(c) <= free;
    }
    T* p = nullptr;
    if (room && cudaMalloc(&p, bytes) != cudaSuccess)
        cudaGetLastError();
    if (!p)
    {
        E->refused = count;
        return nullptr;
    }
    E->buf.free();
    E->buf.p = p;
    E->buf.n = count;
    c.rowPlanRoom = plan ? reinterpret_cast<unsigned char*>(p) + matrices : nullptr;
    return p;
}
template float* ElemMatsOrNull<float>(Ctx&, size_t);
template double* ElemMatsOrNull<double>(Ctx&, size_t);

} // namespace nuto_gpu
