// FP32 tangent of linear cells: SimpleAssembler::BuildMatrix (nuto/mechanics/cell/SimpleAssembler.cpp:100-156) of
// MomentumBalance::Hessian0 (nuto/mechanics/integrands/MomentumBalance.h:36-46) and GradientDamage::Hessian0
// (nuto/mechanics/integrands/GradientDamage.h:92-120) for Quad4 and Hex8 cells with the two-point rule, through element
// matrices (k_cell_matrices) that k_rows_from_slabs (rows.cuh) adds into the CSR rows. No atomics: bitwise reproducible.
//
// k_cell_matrices: a warp takes 32 / NIP cells (4 Hex8 cells), (0) lane (cell, node) stages the node data, (A) lane
// (cell, point) evaluates geometry and law into a record in shared memory, (B) lane (cell, a) integrates the slab of its node,
// all blocks (a, b) in registers; its rows leave through shared memory in address order.
// - As in the FP64 form (tangent64.cu) the material tangent has one ratio rho = lambda / mu at all points, so a displacement
//   block is rho S + S^T + tr(S) I with S = sum of mu w g_a g_b^T; the (disp, eeq) and (eeq, eeq) rows are transposed
//   interpolations (sumfac.cuh). Two neighbours b share a packed FP32 multiply-add (fma.rn.f32x2): the node gradients lie
//   component-major in the record, so that one 16-byte load gives two such pairs.
// - Bound by the shared-memory data path (70 % of its wavefronts at 48^3; a 16-byte load of a warp is four, broadcast or not),
//   then by the 4 KB per Hex8 gradient-damage cell that it stores and the row gather reads back. 64^3: 834 us for both
//   kernels with one lane per node pair (each ordered pair with its own lambda and mu sums), 622 us now; 17^3 31 -> 19 us;
//   200^2 Quad4 elastic 31 -> 15 us. Storing rows with 32-byte stores straight from the lanes: 687 us.
//
// Branch decisions of the law are those of the history update and the FP64 tangent: the nonlocal equivalent strain at a point
// is formed in FP32 with an error bound, and where the bound does not separate it from the history kappa or from kappa0 it is
// recomputed in FP64 in the order of k_history, so a converged loading point, whose kappa is that very value, is loading here.
// (The residual forms it sum-factorised, with other last bits; it takes the larger of the two values, which has no branch.)
// Everything else is FP32.
#include "rows.cuh"
#include "sumfac.cuh"

#include <algorithm>
#include <type_traits>

namespace nuto_gpu
{

namespace
{

struct FusedArgs
{
    int64_t nCells, nDofs, nNodesD, nNodesE;
    int64_t cellFirst, cellLast; // cells of this launch
    const int32_t* connD;        // planar [n][cell]
    const int32_t* connE;
    const int64_t* gdofD; // per node: combined index of component 0
    const int64_t* gdofE;
    const float* relX;    // planar [(n * DIM + d)][cell]: X_n - X_0
    const double* kappa;  // [cell][ip]
    const double* escale; // per-cell Young's modulus factor (nullptr: 1)
    const double* tabN;   // nIp x nd
    const double* tabDN;  // nIp x nd x 3
    const double* tabW;   // nIp
    // the law's parameters in FP32, converted on the host: a conversion is an FP64-pipe instruction (converting u on the
    // integer pipe as well cost more instructions than it saved: 648 against 622 us at 64^3)
    float rho, C33, lamD, muD, m2G, kappa0, alpha, beta, c;
    float K1, K2, nu; // ModifiedMisesStrainNorm
    int planeState;
};

template <int DIM, int KIND>
struct CellShape
{
    static constexpr bool GD = KIND == NUTO_GPU_GRADIENT_DAMAGE;
    static constexpr int nd = SumFac<DIM>::nd, nip = nd;
    static constexpr int cpw = 32 / nip; // cells per warp: one lane per (cell, node) and per (cell, point)
    static constexpr int vd = DIM == 2 ? 3 : 6;
    // record of a point (floats): the node gradients, component-major [d][b]; gradient damage: Q_b = -B_b^T t, likewise, the
    // Voigt vector of P, the eeq-gradient coupling vector, w, c g w; mu w last
    static constexpr int oG = 0, oQ = nd * DIM, oS = 2 * nd * DIM, oC = oS + vd, oW = oC + DIM;
    static constexpr int oMu = GD ? oW + 2 : nd * DIM;
    // rows of an odd number of 16-byte groups, cells offset by one more group: the 8 lanes of a quarter warp that write their
    // point's record, and the lanes of different cells that read one, touch distinct banks
    static constexpr int groups = (oMu + 1 + 3) / 4;
    static constexpr int rec = (groups | 1) * 4;
    static constexpr int cell = nip * rec + 4;
    static constexpr int nodeF = cpw * nd * 8;          // coordinates + eeq and displacements, 2 float4 per (cell, node)
    static constexpr int eF = GD ? cpw * nd * 2 : 0;    // eeq in FP64
    // (dN/dxi, N) per point and node (rows padded by one entry: the lanes of a cell read the rows of different points), weights
    static constexpr int tabRow = nd + 1;
    static constexpr int tabF = nip * tabRow * 4 + (nip + 3) / 4 * 4;
    // staging of one row of every lane's slab: the rows leave as whole 16-byte pieces in address order
    static constexpr int nc = Slab<DIM, nd, GD>::nc;
    static constexpr int stRow = (nc / 4 | 1) * 4;
    static constexpr int stF = 32 * stRow > nodeF + eF ? 32 * stRow : nodeF + eF; // in the place of the node data
    static constexpr int perWarp = stF + cpw * cell;
    static constexpr size_t smem(int W)
    {
        return (static_cast<size_t>(W) * perWarp + tabF) * sizeof(float);
    }
    static_assert(nodeF % 4 == 0 && eF % 4 == 0 && perWarp % 4 == 0 && tabF % 4 == 0, "16-byte regions");
};

// ---- packed FP32 pairs ---------------------------------------------------------------------------------------------
using F2 = unsigned long long;
__device__ __forceinline__ F2 Pk(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void Unpk(F2 r, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ F2 Fma2(F2 a, F2 b, F2 c)
{
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ F2 Add2(F2 a, F2 b)
{
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Geometry, strain and law at integration point q of cell e from the cell's node data: X (coordinates relative to
// the first node, eeq value in .w), U (displacements), E64 (eeq values in FP64, for the branch decisions); T the
// (dN/dxi, N) table row of q and w its weight. Writes the point's record (CellShape). The loading/unloading and damage
// branches are the FP64 tangent's (decided in FP32 where the error bound of eeq separates the operands, else in FP64 as that
// tangent forms eeq: same order, FP64 shape values tabN).
template <int DIM, int KIND>
__device__ __forceinline__ void PointRecord(const FusedArgs& A, const LawParams& L, const float4* T, float w,
                                            const float4* X, const float4* U, const double* E64, int q, int64_t e,
                                            float* rec)
{
    using C = CellShape<DIM, KIND>;
    constexpr bool GD = C::GD;
    constexpr int ND = C::nd, NIP = C::nip, VD = C::vd;
    const int64_t n = A.nCells;
    (void)n;
    float J[DIM][DIM];
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
        for (int j = 0; j < DIM; ++j)
            J[i][j] = 0.f;
#pragma unroll
    for (int nd = 0; nd < ND; ++nd)
    {
        const float4 x = X[nd], t = T[nd];
        const float xv[3] = {x.x, x.y, x.z}, tv[3] = {t.x, t.y, t.z};
#pragma unroll
        for (int i = 0; i < DIM; ++i)
#pragma unroll
            for (int j = 0; j < DIM; ++j)
                J[i][j] += xv[i] * tv[j];
    }
    float det, inv[DIM][DIM];
    if (DIM == 2)
    {
        det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
        const float id = 1.f / det;
        inv[0][0] = J[1][1] * id;
        inv[0][1] = -J[0][1] * id;
        inv[1][0] = -J[1][0] * id;
        inv[1][1] = J[0][0] * id;
    }
    else
    {
        const float c00 = J[1][1] * J[2 % DIM][2 % DIM] - J[1][2 % DIM] * J[2 % DIM][1];
        const float c10 = J[1][2 % DIM] * J[2 % DIM][0] - J[1][0] * J[2 % DIM][2 % DIM];
        const float c20 = J[1][0] * J[2 % DIM][1] - J[1][1] * J[2 % DIM][0];
        det = J[0][0] * c00 + J[0][1] * c10 + J[0][2 % DIM] * c20;
        const float id = 1.f / det;
        inv[0][0] = c00 * id;
        inv[1][0] = c10 * id;
        inv[2 % DIM][0] = c20 * id;
        inv[0][1] = (J[0][2 % DIM] * J[2 % DIM][1] - J[0][1] * J[2 % DIM][2 % DIM]) * id;
        inv[1][1] = (J[0][0] * J[2 % DIM][2 % DIM] - J[0][2 % DIM] * J[2 % DIM][0]) * id;
        inv[2 % DIM][1] = (J[0][1] * J[2 % DIM][0] - J[0][0] * J[2 % DIM][1]) * id;
        inv[0][2 % DIM] = (J[0][1] * J[1][2 % DIM] - J[0][2 % DIM] * J[1][1]) * id;
        inv[1][2 % DIM] = (J[0][2 % DIM] * J[1][0] - J[0][0] * J[1][2 % DIM]) * id;
        inv[2 % DIM][2 % DIM] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * id;
    }
    const float wdj = w * det;
    // per-cell Young's modulus factor: scales the material tangent and dsigma/domega
    const float wdjE = A.escale ? wdj * static_cast<float>(A.escale[e]) : wdj;
    float g[DIM][ND], H[DIM][DIM], ge[DIM];
    float eeq = 0.f, eabs = 0.f;
#pragma unroll
    for (int i = 0; i < DIM; ++i)
    {
        ge[i] = 0.f;
#pragma unroll
        for (int j = 0; j < DIM; ++j)
            H[i][j] = 0.f;
    }
#pragma unroll
    for (int nd = 0; nd < ND; ++nd)
    {
        const float4 t = T[nd];
        const float tv[3] = {t.x, t.y, t.z};
#pragma unroll
        for (int k = 0; k < DIM; ++k)
        {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < DIM; ++j)
                s += tv[j] * inv[j][k];
            g[k][nd] = s;
        }
        if (GD)
        {
            const float4 uv = U[nd];
            const float uc[3] = {uv.x, uv.y, uv.z};
#pragma unroll
            for (int c = 0; c < DIM; ++c)
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    H[c][d] += uc[c] * g[d][nd];
            const float ev = X[nd].w;
            eeq += t.w * ev;
            eabs += fabsf(t.w * ev);
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                ge[d] += ev * g[d][nd];
        }
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
        for (int b = 0; b < ND; b += 4)
            *reinterpret_cast<float4*>(rec + C::oG + d * ND + b) = make_float4(g[d][b], g[d][b + 1], g[d][b + 2], g[d][b + 3]);
    if (!GD)
    {
        rec[C::oMu] = A.C33 * wdjE; // LinearElastic: C33 = mu, C12 = lambda = rho mu
        return;
    }
    float eps[VD];
    StrainFromH<float, DIM>(H, eps);
    const double kh64 = A.kappa[NG_IDX(e * NIP + q, n * NIP, 55)];
    const float kh = static_cast<float>(kh64);
    const float bound = 1.0e-6f * eabs + 1.0e-30f;
    double e64 = 0.;
    float kapLoad = eeq;
    bool have64 = false;
    auto eeq64 = [&]() {
        if (!have64)
        {
            double s = 0.;
            for (int nd = 0; nd < ND; ++nd)
                s += A.tabN[q * ND + nd] * E64[nd];
            e64 = s;
            kapLoad = static_cast<float>(s);
            have64 = true;
        }
        return e64;
    };
    bool loading;
    if (fabsf(eeq - kh) > bound + 1.0e-7f * fabsf(kh))
        loading = eeq >= kh;
    else
        loading = eeq64() >= kh64;
    bool damaged;
    const float k0f = A.kappa0;
    if (!loading)
        damaged = fabsf(kh - k0f) > 2.0e-7f * k0f ? kh >= k0f : kh64 >= L.kappa0; // FP64 where the rounding could decide
    else if (fabsf(eeq - k0f) > bound + 1.0e-7f * k0f)
        damaged = eeq >= k0f;
    else
        damaged = eeq64() >= L.kappa0;
    const float kap = loading ? kapLoad : kh;
    float phi = 1.f, dOdK = 0.f; // 1 - omega and domega/dkappa
    if (damaged)
    {
        // DamageLawExponential (DamageLawExponential.h:40-52) above kappa0
        const float al = A.alpha, be = A.beta;
        const float ex = expf(be * (k0f - kap));
        const float r = k0f / kap;
        phi = r * (1.f - al + al * ex);
        dOdK = loading ? r * ((1.f / kap + be) * al * ex + (1.f - al) / kap) : 0.f;
    }
    float gI = 1.f, dgdw = 0.f;
    if (L.interaction != NUTO_GPU_INTERACTION_CONSTANT)
    {
        gI = InteractionFactor<float>(L, 1.f - phi);
        dgdw = InteractionDerivative<float>(L, 1.f - phi);
    }
    // the factors of the sum-factorised transposes (sumfac.cuh) go into what they transform: P and the (eeq, eeq) vector
    constexpr float vs = static_cast<float>(SumFac<DIM>::valScale);
    // (disp, eeq): B^T (dsigma/domega w' k') N with dsigma/domega = -(lambda tr + 2 mu eps)
    float tr = eps[0] + eps[1];
    if (DIM == 3)
        tr += eps[2];
    const float f = -vs * dOdK * wdjE, t = A.lamD * tr, fm = f * A.muD;
#pragma unroll
    for (int v = 0; v < VD; ++v)
        rec[C::oS + v] = v < DIM ? f * (A.m2G * eps[v] + t) : fm * eps[v];
    const float c = A.c;
    const float sc = vs * c * dgdw * dOdK * wdj;
#pragma unroll
    for (int d = 0; d < DIM; ++d)
        rec[C::oC + d] = sc * ge[d];
    rec[C::oW] = vs * wdj;
    rec[C::oW + 1] = c * gI * wdj;
    rec[C::oMu] = A.muD * phi * wdjE;
    // (eeq, disp): -N^T (deps_eq/deps)^T B
    float dn[VD];
    MisesDerivative<float, DIM>(A, eps, dn);
#pragma unroll
    for (int v = 0; v < VD; ++v)
        dn[v] *= -wdj;
#pragma unroll
    for (int b0 = 0; b0 < ND; b0 += 4)
    {
        float Q[4][DIM];
#pragma unroll
        for (int b = 0; b < 4; ++b)
        {
            float gb[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                gb[d] = g[d][b0 + b];
            BtS<float, DIM>(gb, dn, Q[b]);
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d)
            *reinterpret_cast<float4*>(rec + C::oQ + d * ND + b0) = make_float4(Q[0][d], Q[1][d], Q[2][d], Q[3][d]);
    }
}

// RESIDENT: a grid of resident blocks walks the cells, else one pass per warp
template <int DIM, int KIND, int W, bool RESIDENT>
__global__ void __launch_bounds__(W * 32, 16 / W) k_cell_matrices(FusedArgs A, LawParams L, const double* __restrict__ u,
                                                                  float* __restrict__ em)
{
    using C = CellShape<DIM, KIND>;
    using SL = Slab<DIM, C::nd, C::GD>;
    constexpr bool GD = C::GD;
    constexpr int ND = C::nd, NIP = C::nip, CPW = C::cpw, NP = ND / 2;
    constexpr int NC = SL::nc;
    extern __shared__ __align__(16) float smL[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4* sT = reinterpret_cast<float4*>(smL); // [NIP][tabRow]
    float* sWq = smL + NIP * C::tabRow * 4;      // [NIP]
    float* base = smL + C::tabF + wid * C::perWarp;
    float4* sX = reinterpret_cast<float4*>(base);             // [CPW][ND]
    float4* sU = sX + CPW * ND;                               // [CPW][ND]
    double* sE = reinterpret_cast<double*>(base + C::nodeF);  // [CPW][ND]
    float* sStage = base;                                     // [32][stRow], once the node data are used up
    float* sR = base + C::stF;                                // [CPW] cells of NIP records
    for (int i = threadIdx.x; i < NIP * ND; i += blockDim.x)
    {
        const int q = i / ND, nd = i % ND;
        const double* d = A.tabDN + (q * ND + nd) * 3;
        sT[q * C::tabRow + nd] = make_float4(static_cast<float>(d[0]), static_cast<float>(d[1]), DIM == 3 ? static_cast<float>(d[2]) : 0.f,
                                                 static_cast<float>(A.tabN[q * ND + nd]));
    }
    for (int i = threadIdx.x; i < NIP; i += blockDim.x)
        sWq[i] = static_cast<float>(A.tabW[i]);
    __syncthreads();
    const int64_t n = A.nCells, last = A.cellLast;
    const int64_t stride = RESIDENT ? static_cast<int64_t>(gridDim.x) * W * CPW : n;
    // the warp's own cells: only warp-level synchronisation follows
    for (int64_t c0 = A.cellFirst + (static_cast<int64_t>(blockIdx.x) * W + wid) * CPW; c0 < last; c0 += stride)
    {
        // (0) lane (cell slot, node): the node data; (A) lane (cell slot, point): geometry and law
        const int cl = lane / ND, ia = lane % ND;
        const int64_t e = c0 + cl;
        if (e < last)
        {
            const int32_t nD = static_cast<int32_t>(NG_IDX(A.connD[static_cast<int64_t>(ia) * n + e], A.nNodesD, 80));
            const int64_t gd = A.gdofD[nD];
            float x[3] = {0.f, 0.f, 0.f}, v[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int d = 0; d < DIM; ++d)
            {
                x[d] = A.relX[(static_cast<int64_t>(ia) * DIM + d) * n + e];
                if (GD)
                    v[d] = static_cast<float>(u[NG_IDX(gd + d, A.nDofs, 81)]);
            }
            float ev = 0.f;
            if (GD)
            {
                const int32_t nE = static_cast<int32_t>(NG_IDX(A.connE[static_cast<int64_t>(ia) * n + e], A.nNodesE, 82));
                const double e64 = u[NG_IDX(A.gdofE[nE], A.nDofs, 83)];
                sE[cl * ND + ia] = e64;
                ev = static_cast<float>(e64);
            }
            sX[cl * ND + ia] = make_float4(x[0], x[1], x[2], ev);
            sU[cl * ND + ia] = make_float4(v[0], v[1], v[2], 0.f);
        }
        __syncwarp();
        if (e < last)
            PointRecord<DIM, KIND>(A, L, sT + ia * C::tabRow, sWq[ia], sX + cl * ND, sU + cl * ND, GD ? sE + cl * ND : nullptr, ia,
                                   e, sR + cl * C::cell + ia * C::rec);
        __syncwarp();
        // (B) lane (cell slot, a): the slab of a, row by row through the staging rows
        const bool on = e < last;
        float* R = sR + cl * C::cell;
        float4* st = reinterpret_cast<float4*>(sStage + lane * C::stRow);
        auto flush = [&](int k) {
            __syncwarp();
            constexpr int P4 = NC / 4; // pieces per row
            for (int i = lane; i < 32 * P4; i += 32)
            {
                const int row = i / P4, j = i % P4;
                const int64_t er = c0 + row / ND;
                if (er < last)
                    *reinterpret_cast<float4*>(em + (NG_IDX(er, n, 84) * ND + row % ND) * SL::size + k * NC + 4 * j) =
                            *reinterpret_cast<const float4*>(sStage + row * C::stRow + 4 * j);
            }
            __syncwarp();
        };
        if constexpr (GD)
        {
            // the coupling rows: eu[l][b] = sum of N_a Q_b; dd[b] = sum of c g w (g_a . g_b); and the values over the
            // points that the transposed interpolation turns into the (disp, eeq) rows and the (eeq, eeq) row
            float f[DIM + 1][NIP], o[ND];
            if (on)
            {
                F2 eu[DIM][NP], dd[NP];
#pragma unroll
                for (int p = 0; p < NP; ++p)
                {
                    dd[p] = 0ull;
#pragma unroll
                    for (int l = 0; l < DIM; ++l)
                        eu[l][p] = 0ull;
                }
#pragma unroll
                for (int q = 0; q < NIP; ++q)
                {
                    const float* r = R + q * C::rec;
                    const float Na = sT[q * C::tabRow + ia].w, cgw = r[C::oW + 1];
                    float ga[DIM], sv[C::vd], P[DIM];
                    F2 cg[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                    {
                        ga[d] = r[C::oG + d * ND + ia];
                        cg[d] = Pk(cgw * ga[d], cgw * ga[d]);
                    }
#pragma unroll
                    for (int v = 0; v < C::vd; ++v)
                        sv[v] = r[C::oS + v];
                    BtS<float, DIM>(ga, sv, P);
                    float z = r[C::oW] * Na;
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                    {
                        f[d][q] = P[d];
                        z += r[C::oC + d] * ga[d];
                    }
                    f[DIM][q] = z;
                    const F2 na2 = Pk(Na, Na);
#pragma unroll
                    for (int l = 0; l < DIM; ++l)
#pragma unroll
                        for (int b = 0; b < ND; b += 4)
                        {
                            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(r + C::oQ + l * ND + b);
                            eu[l][b / 2] = Fma2(na2, v.x, eu[l][b / 2]);
                            eu[l][b / 2 + 1] = Fma2(na2, v.y, eu[l][b / 2 + 1]);
                            const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(r + C::oG + l * ND + b);
                            dd[b / 2] = Fma2(cg[l], g.x, dd[b / 2]);
                            dd[b / 2 + 1] = Fma2(cg[l], g.y, dd[b / 2 + 1]);
                        }
                }
                float row[NC];
#pragma unroll
                for (int l = 0; l < DIM; ++l)
#pragma unroll
                    for (int p = 0; p < NP; ++p)
                        Unpk(eu[l][p], row[(2 * p) * DIM + l], row[(2 * p + 1) * DIM + l]);
                SfValuesToNodes<float, DIM>(f[DIM], o);
#pragma unroll
                for (int p = 0; p < NP; ++p)
                {
                    float d0, d1;
                    Unpk(dd[p], d0, d1);
                    row[ND * DIM + 2 * p] = o[2 * p] + d0;
                    row[ND * DIM + 2 * p + 1] = o[2 * p + 1] + d1;
                }
#pragma unroll
                for (int j = 0; j < NC / 4; ++j)
                    st[j] = make_float4(row[4 * j], row[4 * j + 1], row[4 * j + 2], row[4 * j + 3]);
            }
            flush(DIM);
            // the (disp, eeq) rows wait in the place of the lane's own record's Q (no lane reads Q any more)
            if (on)
            {
#pragma unroll
                for (int k = 0; k < DIM; ++k)
                {
                    SfValuesToNodes<float, DIM>(f[k], o);
#pragma unroll
                    for (int b = 0; b < ND; b += 4)
                        *reinterpret_cast<float4*>(R + ia * C::rec + C::oQ + k * ND + b) =
                                make_float4(o[b], o[b + 1], o[b + 2], o[b + 3]);
                }
            }
        }
        F2 s[DIM][DIM][NP];
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int k = 0; k < DIM; ++k)
#pragma unroll
                for (int l = 0; l < DIM; ++l)
                    s[k][l][p] = 0ull;
        if (on)
        {
#pragma unroll 1
            for (int q = 0; q < NIP; ++q)
            {
                const float* r = R + q * C::rec;
                const float muw = r[C::oMu];
                F2 m[DIM];
#pragma unroll
                for (int k = 0; k < DIM; ++k)
                {
                    const float mk = muw * r[C::oG + k * ND + ia];
                    m[k] = Pk(mk, mk);
                }
#pragma unroll
                for (int b = 0; b < ND; b += 4)
                {
                    F2 gb[DIM][2];
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                    {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(r + C::oG + d * ND + b);
                        gb[d][0] = v.x;
                        gb[d][1] = v.y;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int k = 0; k < DIM; ++k)
#pragma unroll
                            for (int l = 0; l < DIM; ++l)
                                s[k][l][b / 2 + h] = Fma2(m[k], gb[l][h], s[k][l][b / 2 + h]);
                }
            }
        }
        const F2 rho2 = Pk(A.rho, A.rho);
        F2 tr[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p)
        {
            tr[p] = Add2(s[0][0][p], s[1][1][p]);
            if (DIM == 3)
                tr[p] = Add2(tr[p], s[DIM - 1][DIM - 1][p]);
        }
#pragma unroll
        for (int k = 0; k < DIM; ++k)
        {
            float row[ND * DIM];
#pragma unroll
            for (int l = 0; l < DIM; ++l)
#pragma unroll
                for (int p = 0; p < NP; ++p)
                {
                    const F2 v = Fma2(rho2, s[k][l][p], k == l ? Add2(s[l][k][p], tr[p]) : s[l][k][p]);
                    Unpk(v, row[(2 * p) * DIM + l], row[(2 * p + 1) * DIM + l]);
                }
#pragma unroll
            for (int j = 0; j < ND * DIM / 4; ++j)
                st[j] = make_float4(row[4 * j], row[4 * j + 1], row[4 * j + 2], row[4 * j + 3]);
            if (GD && on)
            {
#pragma unroll
                for (int b = 0; b < ND; b += 4)
                    st[(ND * DIM + b) / 4] = *reinterpret_cast<const float4*>(R + ia * C::rec + C::oQ + k * ND + b);
            }
            flush(k);
        }
        if (RESIDENT)
            __syncwarp(); // the next pass rewrites the node data and records
    }
}

// planar [(n * dim + d)][cell]: the difference of the node's and the cell's first node's coordinates, formed in FP64
__global__ void __launch_bounds__(256) k_relative_coordinates(int64_t nCells, int nge, int dim, int64_t nValues,
                                                              const double* __restrict__ coords,
                                                              const int32_t* __restrict__ connT, float* __restrict__ rel)
{
    const int64_t e = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (e >= nCells)
        return;
    const int64_t first = static_cast<int64_t>(connT[e]) * dim;
    (void)nValues; // extent of the checked indices
    for (int nd = 0; nd < nge; ++nd)
    {
        const int64_t node = static_cast<int64_t>(connT[nd * nCells + e]) * dim;
        for (int d = 0; d < dim; ++d)
            rel[(static_cast<int64_t>(nd) * dim + d) * nCells + e] =
                    static_cast<float>(coords[NG_IDX(node + d, nValues, 85)] - coords[NG_IDX(first + d, nValues, 85)]);
    }
}

} // namespace

// FP32 coordinates of every cell's nodes relative to its first node (planar [(n * dim + d)][cell]), formed in FP64
// once per mesh: the Jacobian of the FP32 tangent then sees differences of the size of the cell instead of FP32
// absolute coordinates
void BuildRelativeCoordinates(Ctx& c)
{
    c.dRelX.alloc(static_cast<size_t>(c.nge) * c.dim * c.nCells);
    k_relative_coordinates<<<static_cast<unsigned>((c.nCells + 255) / 256), 256, 0, c.stream>>>(
            c.nCells, c.nge, c.dim, static_cast<int64_t>(c.dCoords.n), c.dCoords.p, c.dGeoConnT.p, c.dRelX.p);
    AfterLaunch(c, "k_relative_coordinates");
}

bool FusedTangentSupported(Ctx& c)
{
    if (c.fusedMode >= 0)
        return c.fusedMode == 1;
    c.fusedMode = 0;
    const Slot& D = c.slots[c.prm.disp_slot];
    const bool gd = c.prm.kind == NUTO_GPU_GRADIENT_DAMAGE;
    // linear cells whose coordinate and displacement elements coincide, LinearElastic or GradientDamage with FULL
    // damage application (UNILATERAL switches the volumetric damage on the sign of the volumetric strain, a branch
    // that FP32 cannot decide like FP64 near zero), 2x2 / 2x2x2 Gauss points
    const bool cells = (c.dim == 2 && c.nge == 4 && D.nen == 4 && c.ip.nIp == 4) ||
                       (c.dim == 3 && c.nge == 8 && D.nen == 8 && c.ip.nIp == 8);
    const bool law = c.prm.kind == NUTO_GPU_MB_LINEAR_ELASTIC ||
                     (gd && c.prm.damage_application == NUTO_GPU_DAMAGE_FULL);
    if (!cells || !law)
        return false;
    // every row of a displacement node (and of its eeq node) fits the row buffer
    const int eS = gd ? c.prm.eeq_slot : c.prm.disp_slot;
    for (int s : {c.prm.disp_slot, eS})
    {
        if (c.maxRowLen <= kRowsCap)
            break; // as on every lattice: no scan
        const Slot& S = c.slots[s];
        for (int64_t i = 0; i < S.nNodes; ++i)
            for (int k = 0; k < S.ncomp; ++k)
            {
                const int64_t r = S.offset + S.dof0[i] + k;
                if (c.hRowPtr[r + 1] - c.hRowPtr[r] > kRowsCap)
                    return false;
            }
    }
    c.fusedMode = 1;
    return true;
}

// cellChunkEnd[k]: one past the last cell with a node of the first k + 1 node chunks
static void EnsureCellChunks(Ctx& c, const Slot& D, int chunks)
{
    if (static_cast<int>(c.cellChunkEnd.size()) == chunks)
        return;
    std::vector<int64_t> end(chunks, 0);
    for (int64_t e = 0; e < c.nCells; ++e)
    {
        int64_t node = D.nNodes;
        for (int n = 0; n < D.nen; ++n)
            node = std::min<int64_t>(node, D.conn[e * D.nen + n]);
        int ch = static_cast<int>(node * chunks / D.nNodes); // or the chunk behind it, where the bounds round down
        while (ch > 0 && node < D.nNodes * ch / chunks)
            --ch;
        while (ch + 1 < chunks && node >= D.nNodes * (ch + 1) / chunks)
            ++ch;
        end[ch] = e + 1;
    }
    for (int k = 1; k < chunks; ++k)
        end[k] = std::max(end[k], end[k - 1]);
    c.cellChunkEnd = std::move(end);
}

bool LaunchTangentFused(Ctx& c, const double* u, float* vals)
{
    const int dS = c.prm.disp_slot;
    const bool gd = c.prm.kind == NUTO_GPU_GRADIENT_DAMAGE;
    const int eS = gd ? c.prm.eeq_slot : dS;
    const Slot& D = c.slots[dS];
    const size_t slab = c.dim == 3 ? (gd ? Slab<3, 8, true>::size : Slab<3, 8, false>::size)
                                   : (gd ? Slab<2, 4, true>::size : Slab<2, 4, false>::size);
    float* em = ElemMatsOrNull<float>(c, static_cast<size_t>(c.nCells) * D.nen * slab);
    if (!em)
        return false;
    if (c.dRelX.n == 0)
        BuildRelativeCoordinates(c);
    FusedArgs A{};
    A.nCells = c.nCells;
    A.nDofs = c.nDofs;
    A.nNodesD = D.nNodes;
    A.nNodesE = c.slots[eS].nNodes;
    A.connD = D.dConnT.p;
    A.connE = c.slots[eS].dConnT.p;
    A.gdofD = D.dGdof.p;
    A.gdofE = c.slots[eS].dGdof.p;
    A.relX = c.dRelX.p;
    A.kappa = c.dKappa.p;
    A.escale = c.dEScale.n ? c.dEScale.p : nullptr;
    A.tabN = c.dTables.p + c.tabN[D.interp];
    A.tabDN = c.dTables.p + c.tabDN[D.interp];
    A.tabW = c.dTables.p + c.tabW;
    const LawParams& L = c.law;
    const double mu0 = gd ? L.muD : L.C33;
    A.rho = static_cast<float>(mu0 != 0. ? (gd ? L.lamD : L.C12) / mu0 : 0.);
    A.C33 = static_cast<float>(L.C33);
    A.lamD = static_cast<float>(L.lamD);
    A.muD = static_cast<float>(L.muD);
    A.m2G = static_cast<float>(L.m2G);
    A.kappa0 = static_cast<float>(L.kappa0);
    A.alpha = static_cast<float>(L.alpha);
    A.beta = static_cast<float>(L.beta);
    A.c = static_cast<float>(L.c);
    A.K1 = static_cast<float>(L.K1);
    A.K2 = static_cast<float>(L.K2);
    A.nu = static_cast<float>(L.nu);
    A.planeState = L.planeState;
    const RowPlanArgs plan = EnsureRowPlan(c);
    if (c.slots.size() > static_cast<size_t>(gd ? 2 : 1)) // rows of slots that the integrand does not touch
        NG_CUDA(cudaMemsetAsync(vals, 0, c.nnz * sizeof(float), c.stream));
    // one assembly with W warps per block; form 1: a grid of resident blocks for the cell kernel
    auto assemble = [&](int W, int form) {
        auto run = [&](auto dim, auto kind, auto warps) {
            constexpr int DIM = decltype(dim)::value, KIND = decltype(kind)::value, WW = decltype(warps)::value;
            using C = CellShape<DIM, KIND>;
            constexpr size_t smem = C::smem(WW);
            auto cells = [&](auto kern, bool resident) {
                if (smem > 48 * 1024)
                    NG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(smem)));
                constexpr int64_t perBlock = static_cast<int64_t>(WW) * C::cpw;
                int64_t blocks = (A.cellLast - A.cellFirst + perBlock - 1) / perBlock;
                if (resident)
                {
                    int perSm = 0;
                    NG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, WW * 32, smem));
                    blocks = std::max<int64_t>(1, std::min<int64_t>(blocks, static_cast<int64_t>(perSm) * c.smCount));
                }
                NG_CUDA(LaunchEx(false, c.carveout, kern, dim3(static_cast<unsigned>(blocks)), dim3(WW * 32), smem, c.stream, A,
                                 c.law, u, em));
                AfterLaunch(c, "k_cell_matrices");
                c.stats.kernel_launches += 1;
            };
            // in node chunks when a caller hooks into them: the cells that a chunk's rows are the first to need, then its
            // rows, which are complete when their launch is
            const int chunks = c.rowChunks > 1 && c.onRowChunk ? c.rowChunks : 1;
            if (chunks > 1)
                EnsureCellChunks(c, D, chunks);
            for (int ch = 0; ch < chunks; ++ch)
            {
                const int64_t a0 = D.nNodes * ch / chunks, a1 = D.nNodes * (ch + 1) / chunks;
                A.cellFirst = ch > 0 ? c.cellChunkEnd[ch - 1] : 0;
                A.cellLast = chunks > 1 ? c.cellChunkEnd[ch] : c.nCells;
                if (A.cellLast > A.cellFirst)
                {
                    if (form == 1)
                        cells(k_cell_matrices<DIM, KIND, WW, true>, true);
                    else
                        cells(k_cell_matrices<DIM, KIND, WW, false>, false);
                }
                LaunchRows<float, DIM, C::nd, C::GD, WW>(c, plan, a0, a1, em, vals);
                if (chunks > 1)
                {
                    c.onRowChunk(a0, a1);
                    c.rowChunksDone++;
                }
            }
        };
        auto withWarps = [&](auto dim, auto kind) {
            if (W == 2)
                run(dim, kind, std::integral_constant<int, 2>{});
            else if (W == 8)
                run(dim, kind, std::integral_constant<int, 8>{});
            else
                run(dim, kind, std::integral_constant<int, 4>{});
        };
        using D2 = std::integral_constant<int, 2>;
        using D3 = std::integral_constant<int, 3>;
        using Gd = std::integral_constant<int, NUTO_GPU_GRADIENT_DAMAGE>;
        using El = std::integral_constant<int, NUTO_GPU_MB_LINEAR_ELASTIC>;
        if (c.dim == 3 && gd)
            withWarps(D3{}, Gd{});
        else if (c.dim == 3)
            withWarps(D3{}, El{});
        else if (gd)
            withWarps(D2{}, Gd{});
        else
            withWarps(D2{}, El{});
    };
    // autotuner: the first FP32 tangent of a context (outside any stream capture) assembles once with each candidate
    // shape — 2, 4 and 8 warps per block, and the grid of resident blocks with 2 and 4 — (a warm-up and a timed assembly
    // each; every one writes the same values) and keeps the fastest
    Tuning& T = c.tuning;
    if (T.tangentWarps == 0)
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        NG_CUDA(cudaStreamIsCapturing(c.stream, &cs));
        if (!T.enabled)
            T.tangentWarps = 4;
        else if (cs == cudaStreamCaptureStatusNone)
        {
            const int candW[5] = {2, 4, 8, 2, 4};
            const int candForm[5] = {2, 2, 2, 1, 1};
            cudaEvent_t e0, e1;
            NG_CUDA(cudaEventCreate(&e0));
            NG_CUDA(cudaEventCreate(&e1));
            float best = 0.f;
            int pick = 1;
            for (int k = 0; k < 5; ++k)
            {
                assemble(candW[k], candForm[k]);
                NG_CUDA(cudaEventRecord(e0, c.stream));
                assemble(candW[k], candForm[k]);
                NG_CUDA(cudaEventRecord(e1, c.stream));
                NG_CUDA(cudaEventSynchronize(e1));
                float ms = 0.f;
                NG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                T.tangentMs[k] = ms;
                if (k == 0 || ms < best)
                {
                    best = ms;
                    pick = k;
                }
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            T.tangentMs[5] = T.tangentMs[0];
            T.tangentMs[6] = T.tangentMs[1];
            T.tangentWarps = candW[pick];
            T.tangentForm = candForm[pick];
        }
    }
    assemble(T.tangentWarps ? T.tangentWarps : 4, T.tangentForm);
    return true;
}

} // namespace nuto_gpu
