// Multigrid preconditioner for the Krylov solvers. The reference has no iterative solver on this
// path (it factorises the matrix, EigenSparseSolve.cpp:22-73); this is the GB300-side replacement of that
// factorisation inside the Newton loop.
//
// Structure: one hierarchy per DOF slot (displacements, nonlocal equivalent strains), applied as one block
// Gauss-Seidel sweep in slot order: z_0 = V_0(v_0), z_1 = V_1(v_1 - K_10 z_0). For gradient damage K_10 (the
// dependence of the eeq equation on the local strain) is the strong coupling and K_01 vanishes outside the
// damaging zone, so the sweep is exact there up to the V-cycles.
//
// Hierarchy (host, once per pattern): every level keeps an independent set of the finer level's DOF nodes, taken in node
// order (a node with no kept neighbour is kept), so on a structured mesh about every second one per axis. Axes are coarsened
// while the cells are short along them: neighbours across an axis that is longer than the shortest by more than half do not
// count (the 1 x 1 x 4 beam first coarsens across its short sides). A kept node hands its value on; any other interpolates
// between its (at most 8, the nearest) kept neighbours with weights 1 / distance, which on a lattice is the multilinear
// interpolation. Quadratic cells first drop to their corner nodes with the linear shape functions as weights. Levels stop at
// kCoarsest nodes. Restriction is the transpose; constrained DOFs take part in neither. Against aggregates of the same size with
// piecewise constant transfer, GMRES on a damaged, distorted beam to 1e-13 went from 306 iterations (52 ms) to 96 (18.5 ms) at
// 24^3 in FP32 and from 302 (88 ms) to 57 (18 ms) at 20^3 in FP64; with exact solves of both blocks it takes 25 at 16^3.
// Coarse operators keep the node-block CSR layout, so the node SpMV serves every level; level 0 is a diagonal-block view of
// the tangent itself.
//
// Per tangent (device, in the arithmetic of the tangent: FP32 or FP64): Galerkin coarse values A_c = P^T A P by
// one pass over the finer values, A P in shared memory and the rest with atomics; Jacobi diagonals and Gershgorin
// bounds of D^-1 A per level. Cycle: V(1,2) with Chebyshev-Jacobi smoothing on [lmax / 10, lmax] and a degree-6 Chebyshev solve on the coarsest level. The sweep is a fixed
// linear operator; GMRES uses it in flexible form (stored preconditioned basis) so rounding inside the cycle does
// not limit the attainable residual.
#include "spmv.cuh"

#include <algorithm>
#include <cstdlib>
#include <memory>
#include <cmath>
#include <utility>

namespace nuto_gpu
{

constexpr int kCoarsest = 64; // nodes on the coarsest level
constexpr int kInterp = 8;    // most coarse nodes that a finer node interpolates between
constexpr int kMaxLevels = 12;
constexpr int kPreDegree = 1;
constexpr int kPostDegree = 2;
// Chebyshev degree on the coarsest level, per arithmetic of the cycle: measured on the damaged 64^3 tangent
// (time to a 1e-4 / 1e-7 relative residual), degree 10 made the FP32 cycle 10 % faster than degree 6 and the FP64
// cycle 3 % faster / 7 % slower
template <typename TA>
constexpr int CoarseDegree()
{
    return sizeof(TA) == 4 ? 10 : 6;
}
constexpr float kSmoothRatio = 10.f; // smoothing interval [lmax / ratio, lmax]
constexpr float kCoarseRatio = 30.f;

// vectors and coarse values of one level in the preconditioner's arithmetic TA (FP32 for FP32 tangents, FP64 for
// the plain FP64 path); on level 0 the vectors span the combined system and vals is unused (the tangent is used)
template <typename TA>
struct Num
{
    DBuf<TA> vals, dinv, e, t, d;
    TA* b = nullptr; // coarse levels: right-hand side, a part of Amg::rhs (zeroed once per sweep)
    DBuf<TA> nb; // coarse levels: the values in the padded layout of the level's SpMV
};

// The one-block tail (k_amg_tail) as a dense matrix: its V-cycle is a fixed linear map of at most kTailNodes x 3 values,
// applied once per sweep; column k = the cycle of unit vector k
template <typename TA>
struct TailDense
{
    DBuf<TA> m;    // [k][i]
    DBuf<TA> work; // vectors of the tail levels, one set per column
    int64_t n = 0;
};

// What a level's nodes are, whatever lives on them: neighbour lists and, on coarse levels, the interpolation from them to the
// finer level. Slots on the same nodes (displacements and nonlocal strains of linear cells) share it.
struct LevelNodes
{
    int64_t n = 0;
    std::vector<int64_t> nbrPtr;
    std::vector<int32_t> nbrIdx;
    std::vector<double> coords; // 3 per node
    int maxList = 0;            // longest neighbour list
    // coarse levels
    DBuf<int64_t> dNbrPtr;
    DBuf<int32_t> dNbrIdx;
    DBuf<int32_t> pNode; // kInterp per finer node: nodes of this level, -1 behind the last
    DBuf<float> pWeight; // and their weights
    DBuf<double> pWeight64; // the same values for the FP64 cycle (a conversion is an FP64 instruction), on first use
};

struct AmgLevel
{
    int ncomp = 1;
    std::shared_ptr<LevelNodes> nodes;
    int64_t nNodes = 0;
    int64_t nDofs = 0, nnz = 0;
    // level-0 views address the combined vectors: rows [off, off + nDofs) of the slot
    int64_t off = 0;
    // device structure of coarse levels (level 0 uses the context's pattern)
    DBuf<int64_t> gdof, rowPtr;
    DBuf<int32_t> nbrCol, blk;
    DBuf<int32_t> diagOff;  // per node: offset of the diagonal block in the node's row segment
    DBuf<int64_t> nbBase;   // coarse levels: per node, first value of the node's block in the padded layout
    int64_t nbTotal = 0;
    int nbSeg4 = 0;
    DBuf<uint8_t> zeroMask; // coarse levels have no constrained rows
    // numerics, per arithmetic of the preconditioner (allocated on first use of that arithmetic)
    Num<float> n32;
    Num<double> n64;
    float lmax = 1.f;
    NodeSpmv spmv{};
};

template <typename TA>
static Num<TA>& N(AmgLevel& L);
template <>
Num<float>& N<float>(AmgLevel& L)
{
    return L.n32;
}
template <>
Num<double>& N<double>(AmgLevel& L)
{
    return L.n64;
}

// One sweep (all launches of both V-cycles) captured as a CUDA graph on fixed input/output vectors. The graph is
// recaptured after every set-up (the Chebyshev coefficients are kernel arguments) and the executable graph updated
// in place (same topology), so a sweep costs one launch on the host instead of about 150.
struct SweepGraph
{
    cudaGraphExec_t exec = nullptr;
    uint64_t setup = 0;      // set-up counter the graph was captured for
    const int* st = nullptr; // Krylov state pointer baked into the graph
    int64_t launches = 0;    // kernels per replay
};

struct Amg
{
    int ns = 0;
    std::vector<AmgLevel> h[kMaxSlots];
    DBuf<float> lmaxDev; // all levels of all hierarchies
    std::vector<float> lmaxHost;
    DBuf<float> in32, out32, res32; // combined-length work vectors of the sweep (FP32 cycle)
    DBuf<double> in64, out64, res64; // the same for the FP64 cycle
    DBuf<float> rhs32; // right-hand sides of all coarse levels (Num::b)
    DBuf<double> rhs64;
    TailDense<float> tail32[kMaxSlots];
    TailDense<double> tail64[kMaxSlots];
    bool tailSym = false; // the cycle the tails were formed for
    int prec = 32;                   // arithmetic of the last set-up: that of the tangent values
    const void* fine = nullptr;      // the tangent of the last set-up (level-0 operator)
    const void* setupVals = nullptr;
    uint64_t setupVersion = 0;
    uint64_t setups = 0; // set-ups so far
    bool built = false;
    bool graphs = true;           // NUTO_GPU_GRAPHS=0 launches the sweep kernel by kernel
    SweepGraph graph[2][2];       // [FP64][symmetric]
    ~Amg()
    {
        for (auto& row : graph)
            for (SweepGraph& g : row)
                if (g.exec)
                    cudaGraphExecDestroy(g.exec);
        if (capStream)
            cudaStreamDestroy(capStream);
    }
    bool graphLaunched = false;    // a sweep graph was launched since the hierarchy was built
    std::string graphError; // why graphs were switched off (diagnostics)
    cudaStream_t capStream = nullptr; // private stream for graph capture (the context's may be the legacy stream)
};

template <typename TA>
static DBuf<TA>& Weights(LevelNodes& X)
{
    if constexpr (sizeof(TA) == 4)
        return X.pWeight;
    else
        return X.pWeight64;
}
template <typename TA>
static DBuf<TA>& Rhs(Amg& M)
{
    if constexpr (sizeof(TA) == 4)
        return M.rhs32;
    else
        return M.rhs64;
}
template <typename TA>
static TailDense<TA>& Tail(Amg& M, int slot)
{
    if constexpr (sizeof(TA) == 4)
        return M.tail32[slot];
    else
        return M.tail64[slot];
}

void FreeAmg(Ctx& c)
{
    delete c.amg;
    c.amg = nullptr;
}

// ---- host: hierarchy -------------------------------------------------------------------------------------------
// natural coordinates of the local nodes (InterpolationQuadLinear / BrickLinear / BrickQuadratic order)
static void LocalNodeCoords(int interp, int n, double* xi)
{
    static const double h20[20][3] = {{-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1}, {-1, -1, 1}, {1, -1, 1},
                                      {1, 1, 1},    {-1, 1, 1},  {0, -1, -1}, {1, 0, -1},  {0, 1, -1},  {-1, 0, -1},
                                      {-1, -1, 0},  {1, -1, 0},  {1, 1, 0},   {-1, 1, 0},  {0, -1, 1},  {1, 0, 1},
                                      {0, 1, 1},    {-1, 0, 1}};
    static const double q4[4][2] = {{-1, -1}, {1, -1}, {1, 1}, {-1, 1}};
    if (interp == NUTO_GPU_QUAD4)
    {
        xi[0] = q4[n][0];
        xi[1] = q4[n][1];
        xi[2] = 0;
        return;
    }
    for (int d = 0; d < 3; ++d)
        xi[d] = h20[n][d];
}

// shape functions of the coordinate element (Quad4 / Hex8) at a natural point
static void GeoShape(int geo, const double* xi, double* N)
{
    if (geo == NUTO_GPU_QUAD4)
    {
        const double r = xi[0], s = xi[1];
        N[0] = 0.25 * (1 - r) * (1 - s);
        N[1] = 0.25 * (1 + r) * (1 - s);
        N[2] = 0.25 * (1 + r) * (1 + s);
        N[3] = 0.25 * (1 - r) * (1 + s);
        return;
    }
    const int sg[8][3] = {{-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1},
                          {-1, -1, 1},  {1, -1, 1},  {1, 1, 1},  {-1, 1, 1}};
    for (int i = 0; i < 8; ++i)
        N[i] = 0.125 * (1 + sg[i][0] * xi[0]) * (1 + sg[i][1] * xi[1]) * (1 + sg[i][2] * xi[2]);
}

// per node: offset of the node's own block inside its neighbour segment
static std::vector<int32_t> DiagOffsets(const std::vector<int64_t>& ptr, const std::vector<int32_t>& idx, int ncomp)
{
    const int64_t n = static_cast<int64_t>(ptr.size()) - 1;
    std::vector<int32_t> off(n, 0);
    for (int64_t a = 0; a < n; ++a)
    {
        const int32_t* first = idx.data() + ptr[a];
        const int32_t* last = idx.data() + ptr[a + 1];
        const int32_t* it = std::find(first, last, static_cast<int32_t>(a));
        NG_CHECK(it != last, NUTO_GPU_EINVAL, "a node is missing from its own neighbour list");
        off[a] = static_cast<int32_t>(ncomp * (it - first));
    }
    return off;
}

template <typename T>
static void UploadV(DBuf<T>& buf, const std::vector<T>& h)
{
    buf.alloc(h.size());
    if (!h.empty())
        NG_CUDA(cudaMemcpy(buf.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
}

// single-slot NodeSpmv of a coarse level
static void FillSpmv(AmgLevel& L)
{
    NodeSpmv& A = L.spmv;
    A = NodeSpmv{};
    A.ns = 1;
    A.ncomp[0] = L.ncomp;
    A.nNodes[0] = L.nNodes;
    A.firstWarp[0] = 0;
    A.totalWarps = L.nNodes;
    A.gdof[0] = L.gdof.p;
    A.nbrPtr[0] = L.nodes->dNbrPtr.p;
    A.nbrIdx[0] = L.nodes->dNbrIdx.p;
    A.nbrCol[0] = L.nbrCol.p;
    A.blk[0] = L.blk.p;
    A.nbrTotal[0] = static_cast<int64_t>(L.nodes->dNbrIdx.n);
    A.rowPtr = L.rowPtr.p;
    A.nnz = L.nnz;
    A.nRows = L.nDofs;
}

// diagonal-block view of slot I of the context's tangent
static NodeSpmv SlotView(const Ctx& c, int I)
{
    const int ns = static_cast<int>(c.slots.size());
    const PairMap& M = c.pairs[I * ns + I];
    NodeSpmv A{};
    A.ns = 1;
    A.ncomp[0] = c.slots[I].ncomp;
    A.nNodes[0] = c.slots[I].nNodes;
    A.firstWarp[0] = 0;
    A.totalWarps = c.slots[I].nNodes;
    A.gdof[0] = c.slots[I].dGdof.p;
    A.nbrPtr[0] = M.dNbrPtr.p;
    A.nbrIdx[0] = M.dNbrIdx.p;
    A.nbrCol[0] = M.dNbrCol.p;
    A.blk[0] = M.dBlk.p;
    A.nbrTotal[0] = static_cast<int64_t>(M.dNbrIdx.n);
    A.rowPtr = c.dRowPtr.p;
    A.nnz = c.nnz;
    A.nRows = c.nDofs;
    if (c.nb.total > 0)
    {
        A.nbBase[0] = c.nb.pair[I * ns + I].base.p;
        A.nbOff[0] = c.nb.pair[I * ns + I].off;
        A.nbSeg4 = c.nb.pair[I * ns + I].maxSeg4;
        A.ncMaxRows = c.slots[I].ncomp;
        A.nb32 = c.nb.v32.p;
        A.nb64 = c.nb.v64.p;
        A.nbSrc32 = c.nb.src32;
        A.nbSrc64 = c.nb.src64;
    }
    return A;
}

// axes to coarsen: those shorter than the longest spacing by more than half, or all
static void CoarsenAxes(const double* spacing, int dim, bool* axes)
{
    double mx = 0;
    for (int d = 0; d < dim; ++d)
        mx = std::max(mx, spacing[d]);
    bool any = false;
    for (int d = 0; d < dim; ++d)
        any = any || spacing[d] * 1.5 < mx;
    for (int d = 0; d < dim; ++d)
        axes[d] = !any || spacing[d] * 1.5 < mx;
}

// interpolation of a finer level from the nodes kept: kInterp entries per node
struct Interpolation
{
    int64_t nCoarse = 0;
    std::vector<int32_t> node;
    std::vector<float> weight;
    std::vector<int64_t> kept; // coarse node -> finer node
    void Resize(int64_t n)
    {
        node.assign(n * kInterp, -1);
        weight.assign(n * kInterp, 0.f);
        kept.clear();
    }
};

// neighbours whose distance along an axis that is not coarsened is below half its spacing count
static bool Couples(const LevelNodes& F, int64_t a, int64_t b, int dim, const double* spacing, const bool* axes)
{
    for (int d = 0; d < dim; ++d)
        if (!axes[d] && std::fabs(F.coords[a * 3 + d] - F.coords[b * 3 + d]) >= 0.5 * spacing[d])
            return false;
    return true;
}

// independent set in node order, inverse-distance weights (at most `most` entries per node)
static void KeepNodes(const LevelNodes& F, int dim, const double* spacing, const bool* axes, int most, Interpolation& P)
{
    P.Resize(F.n);
    std::vector<int32_t> coarse(F.n, -1);
    std::vector<char> seen(F.n, 0);
    for (int64_t a = 0; a < F.n; ++a)
    {
        if (seen[a])
            continue;
        coarse[a] = static_cast<int32_t>(P.kept.size());
        P.kept.push_back(a);
        for (int64_t q = F.nbrPtr[a]; q < F.nbrPtr[a + 1]; ++q)
            if (Couples(F, a, F.nbrIdx[q], dim, spacing, axes))
                seen[F.nbrIdx[q]] = 1;
    }
    P.nCoarse = static_cast<int64_t>(P.kept.size());
#pragma omp parallel for schedule(static)
    for (int64_t a = 0; a < F.n; ++a)
    {
        int32_t* pn = P.node.data() + a * kInterp;
        float* pw = P.weight.data() + a * kInterp;
        if (coarse[a] >= 0)
        {
            pn[0] = coarse[a];
            pw[0] = 1.f;
            continue;
        }
        std::pair<double, int32_t> near[kInterp + 1];
        int n = 0;
        for (int64_t q = F.nbrPtr[a]; q < F.nbrPtr[a + 1]; ++q)
        {
            const int32_t b = F.nbrIdx[q];
            if (coarse[b] < 0 || !Couples(F, a, b, dim, spacing, axes))
                continue;
            double d2 = 0;
            for (int d = 0; d < dim; ++d)
                d2 += (F.coords[a * 3 + d] - F.coords[b * 3 + d]) * (F.coords[a * 3 + d] - F.coords[b * 3 + d]);
            int at = n;
            for (; at > 0 && near[at - 1].first > d2; --at)
                near[at] = near[at - 1];
            near[at] = {d2, coarse[b]};
            n = std::min(n + 1, most);
        }
        double sum = 0;
        for (int k = 0; k < n; ++k)
        {
            near[k].first = 1. / std::sqrt(std::max(near[k].first, 1e-30 + 1e-12 * near[n - 1].first));
            sum += near[k].first;
        }
        for (int k = 0; k < n; ++k)
        {
            pn[k] = near[k].second;
            pw[k] = static_cast<float>(near[k].first / sum);
        }
    }
}

// quadratic cells: the corner nodes are kept, the others take the coordinate element's shape functions as weights
static void KeepCorners(const Ctx& c, const Slot& S, Interpolation& P)
{
    P.Resize(S.nNodes);
    std::vector<int32_t> coarse(S.nNodes, -1);
    for (int64_t e = 0; e < c.nCells; ++e)
        for (int g = 0; g < c.nge; ++g)
            coarse[S.conn[e * S.nen + g]] = 0;
    for (int64_t a = 0; a < S.nNodes; ++a)
        if (coarse[a] == 0)
        {
            coarse[a] = static_cast<int32_t>(P.kept.size());
            P.kept.push_back(a);
        }
    P.nCoarse = static_cast<int64_t>(P.kept.size());
    for (int64_t e = 0; e < c.nCells; ++e)
        for (int n = 0; n < S.nen; ++n)
        {
            const int64_t a = S.conn[e * S.nen + n];
            int32_t* pn = P.node.data() + a * kInterp;
            float* pw = P.weight.data() + a * kInterp;
            if (pn[0] >= 0)
                continue;
            if (coarse[a] >= 0)
            {
                pn[0] = coarse[a];
                pw[0] = 1.f;
                continue;
            }
            double xi[3], N[8];
            LocalNodeCoords(S.interp, n, xi);
            GeoShape(c.geoInterp, xi, N);
            int k = 0;
            for (int g = 0; g < c.nge; ++g)
                if (N[g] != 0.)
                {
                    pn[k] = coarse[S.conn[e * S.nen + g]];
                    pw[k++] = static_cast<float>(N[g]);
                }
        }
}

// neighbour lists of the coarse level: i and j are neighbours if P^T A P couples them; false: a list is longer than the
// product supports
static bool CoarseLists(const LevelNodes& F, int ncomp, const Interpolation& P, LevelNodes& C)
{
    std::vector<int64_t> ptr(P.nCoarse + 1, 0);
    for (int32_t i : P.node)
        if (i >= 0)
            ptr[i + 1]++;
    for (int64_t i = 0; i < P.nCoarse; ++i)
        ptr[i + 1] += ptr[i];
    std::vector<int64_t> fill(ptr.begin(), ptr.end() - 1);
    std::vector<int32_t> mem(ptr.back());
    for (int64_t a = 0; a < F.n; ++a)
        for (int k = 0; k < kInterp && P.node[a * kInterp + k] >= 0; ++k)
            mem[fill[P.node[a * kInterp + k]]++] = static_cast<int32_t>(a);
    std::vector<std::vector<int32_t>> lists(P.nCoarse);
#pragma omp parallel
    {
        std::vector<int32_t> mark(P.nCoarse, -1), markFine(F.n, -1);
#pragma omp for schedule(dynamic, 256)
        for (int64_t i = 0; i < P.nCoarse; ++i)
        {
            auto& v = lists[i];
            for (int64_t m = ptr[i]; m < ptr[i + 1]; ++m)
                for (int64_t q = F.nbrPtr[mem[m]]; q < F.nbrPtr[mem[m] + 1]; ++q)
                {
                    const int64_t b = F.nbrIdx[q];
                    if (markFine[b] == i)
                        continue;
                    markFine[b] = static_cast<int32_t>(i);
                    for (int k = 0; k < kInterp && P.node[b * kInterp + k] >= 0; ++k)
                    {
                        const int32_t j = P.node[b * kInterp + k];
                        if (mark[j] != i)
                        {
                            mark[j] = static_cast<int32_t>(i);
                            v.push_back(j);
                        }
                    }
                }
            std::sort(v.begin(), v.end());
        }
    }
    C.nbrPtr.assign(P.nCoarse + 1, 0);
    int64_t longest = 0;
    for (int64_t i = 0; i < P.nCoarse; ++i)
    {
        C.nbrPtr[i + 1] = C.nbrPtr[i] + static_cast<int64_t>(lists[i].size());
        longest = std::max(longest, static_cast<int64_t>(lists[i].size()));
    }
    if (longest * ncomp > kMaxRowLen)
        return false;
    C.maxList = static_cast<int>(longest);
    C.nbrIdx.resize(C.nbrPtr.back());
    for (int64_t i = 0; i < P.nCoarse; ++i)
        std::copy(lists[i].begin(), lists[i].end(), C.nbrIdx.begin() + C.nbrPtr[i]);
    return true;
}

// same: the hierarchy of a slot on the same nodes with at least as many components, or nullptr
static void BuildSlotHierarchy(Ctx& c, int I, const double* ext, std::vector<AmgLevel>& H,
                               const std::vector<AmgLevel>* same)
{
    const int ns = static_cast<int>(c.slots.size());
    const Slot& S = c.slots[I];
    H.clear();
    H.emplace_back();
    {
        AmgLevel& F = H[0];
        F.ncomp = S.ncomp;
        F.nNodes = S.nNodes;
        F.nDofs = S.nDofs;
        F.off = S.offset;
        if (same)
            F.nodes = (*same)[0].nodes;
        else
        {
            F.nodes = std::make_shared<LevelNodes>();
            LevelNodes& X = *F.nodes;
            X.n = S.nNodes;
            X.nbrPtr = c.pairs[I * ns + I].hNbrPtr;
            X.nbrIdx = c.pairs[I * ns + I].hNbrIdx;
            // DOF-node coordinates: the coordinate element interpolated at the node's natural coordinates
            X.coords.assign(S.nNodes * 3, 0.);
            std::vector<double> shape(S.nen * 8);
            for (int n = 0; n < S.nen; ++n)
            {
                double xi[3];
                LocalNodeCoords(S.interp, n, xi);
                GeoShape(c.geoInterp, xi, shape.data() + n * 8);
            }
            std::vector<char> done(S.nNodes, 0);
            for (int64_t e = 0; e < c.nCells; ++e)
                for (int n = 0; n < S.nen; ++n)
                {
                    const int32_t node = S.conn[e * S.nen + n];
                    if (done[node])
                        continue;
                    done[node] = 1;
                    for (int d = 0; d < c.dim; ++d)
                    {
                        double v = 0;
                        for (int g = 0; g < c.nge; ++g)
                            v += shape[n * 8 + g] *
                                 c.hCoords[static_cast<size_t>(c.hGeoConn[e * c.nge + g]) * c.dim + d];
                        X.coords[node * 3 + d] = v;
                    }
                }
        }
        UploadV(F.diagOff, DiagOffsets(F.nodes->nbrPtr, F.nodes->nbrIdx, F.ncomp));
        F.spmv = SlotView(c, I);
    }
    double spacing[3] = {ext[0], ext[1], ext[2]};
    const bool quadratic = S.nen > c.nge;
    for (int level = 1; level < kMaxLevels; ++level)
    {
        AmgLevel& Fi = H[level - 1];
        if (Fi.nNodes <= kCoarsest)
            break;
        AmgLevel C;
        C.ncomp = Fi.ncomp;
        if (same)
        {
            if (static_cast<size_t>(level) >= same->size())
                break;
            C.nodes = (*same)[level].nodes;
        }
        else
        {
            const LevelNodes& FN = *Fi.nodes;
            C.nodes = std::make_shared<LevelNodes>();
            LevelNodes& X = *C.nodes;
            Interpolation P;
            bool axes[3] = {true, true, true}, usable = false;
            if (level == 1 && quadratic)
            {
                KeepCorners(c, S, P);
                usable = CoarseLists(FN, C.ncomp, P, X);
                for (int d = 0; d < c.dim; ++d)
                    axes[d] = false; // corner to corner is one cell extent
            }
            else
            {
                CoarsenAxes(spacing, c.dim, axes);
                // what to try in turn: the chosen axes, all axes, and (where the interpolated stencil is denser than the
                // product supports) the value of the nearest kept node alone
                for (int attempt = 0; attempt < 3 && !usable; ++attempt)
                {
                    if (attempt == 1)
                        for (int d = 0; d < c.dim; ++d)
                            axes[d] = true;
                    KeepNodes(FN, c.dim, spacing, axes, attempt == 2 ? 1 : kInterp, P);
                    usable = P.nCoarse * 5 < FN.n * 4 && CoarseLists(FN, C.ncomp, P, X);
                }
            }
            if (!usable)
                break; // the finer level stays the coarsest
            X.n = P.nCoarse;
            X.coords.resize(X.n * 3);
            for (int64_t i = 0; i < X.n; ++i)
                std::copy_n(FN.coords.begin() + P.kept[i] * 3, 3, X.coords.begin() + i * 3);
            UploadV(X.dNbrPtr, X.nbrPtr);
            UploadV(X.dNbrIdx, X.nbrIdx);
            UploadV(X.pNode, P.node);
            UploadV(X.pWeight, P.weight);
            for (int d = 0; d < c.dim; ++d)
                if (axes[d])
                    spacing[d] *= 2.;
        }
        const std::vector<int64_t>& nbrPtr = C.nodes->nbrPtr;
        const std::vector<int32_t>& nbrIdx = C.nodes->nbrIdx;
        C.nNodes = C.nodes->n;
        // node-block CSR of the coarse level
        C.nDofs = C.nNodes * C.ncomp;
        std::vector<int64_t> rowPtr(C.nDofs + 1, 0), gdof(C.nNodes);
        std::vector<int32_t> blk(C.nNodes, 0);
        for (int64_t A = 0; A < C.nNodes; ++A)
        {
            gdof[A] = A * C.ncomp;
            const int64_t len = C.ncomp * (nbrPtr[A + 1] - nbrPtr[A]);
            for (int k = 0; k < C.ncomp; ++k)
                rowPtr[A * C.ncomp + k + 1] = len;
        }
        for (int64_t r = 0; r < C.nDofs; ++r)
            rowPtr[r + 1] += rowPtr[r];
        C.nnz = rowPtr.back();
        UploadV(C.rowPtr, rowPtr);
        UploadV(C.gdof, gdof);
        UploadV(C.blk, blk);
        {
            std::vector<int32_t> col(nbrIdx.size());
            for (size_t q = 0; q < col.size(); ++q)
                col[q] = nbrIdx[q] * C.ncomp;
            UploadV(C.nbrCol, col);
        }
        UploadV(C.diagOff, DiagOffsets(nbrPtr, nbrIdx, C.ncomp));
        {
            // padded layout of the level: per node ncomp rows of ncomp * nn values, padded to multiples of 4
            std::vector<int64_t> base(C.nNodes);
            int64_t pos = 0;
            int mx = 0;
            for (int64_t A = 0; A < C.nNodes; ++A)
            {
                const int seg4 = static_cast<int>((C.ncomp * (nbrPtr[A + 1] - nbrPtr[A]) + 3) / 4 * 4);
                base[A] = pos;
                pos += static_cast<int64_t>(C.ncomp) * seg4;
                mx = std::max(mx, seg4);
            }
            UploadV(C.nbBase, base);
            C.nbTotal = pos;
            C.nbSeg4 = mx;
        }
        C.zeroMask.alloc(C.nDofs);
        NG_CUDA(cudaMemset(C.zeroMask.p, 0, C.nDofs));
        FillSpmv(C);
        H.push_back(std::move(C));
    }
    H[0].nnz = c.nnz;
}

static void BuildHierarchy(Ctx& c)
{
    Amg& M = *c.amg;
    M.ns = static_cast<int>(c.slots.size());
    // median cell extent per axis (every 7th cell)
    double ext[3] = {1, 1, 1};
    for (int d = 0; d < c.dim; ++d)
    {
        std::vector<double> v;
        for (int64_t e = 0; e < c.nCells; e += 7)
        {
            double lo = 1e300, hi = -1e300;
            for (int g = 0; g < c.nge; ++g)
            {
                const double x = c.hCoords[static_cast<size_t>(c.hGeoConn[e * c.nge + g]) * c.dim + d];
                lo = std::min(lo, x);
                hi = std::max(hi, x);
            }
            v.push_back(hi - lo);
        }
        std::nth_element(v.begin(), v.begin() + v.size() / 2, v.end());
        ext[d] = v[v.size() / 2];
        NG_CHECK(ext[d] > 0, NUTO_GPU_EINVAL, "degenerate cells");
    }
    size_t total = 0;
    for (int I = 0; I < M.ns; ++I)
    {
        // an earlier slot on the same nodes
        const std::vector<AmgLevel>* same = nullptr;
        for (int J = 0; J < I && !same; ++J)
        {
            const Slot &A = c.slots[I], &B = c.slots[J];
            const PairMap &PA = c.pairs[I * M.ns + I], &PB = c.pairs[J * M.ns + J];
            if (A.interp == B.interp && A.nNodes == B.nNodes && A.ncomp <= B.ncomp && A.conn == B.conn &&
                PA.hNbrPtr == PB.hNbrPtr && PA.hNbrIdx == PB.hNbrIdx)
                same = &M.h[J];
        }
        BuildSlotHierarchy(c, I, ext, M.h[I], same);
        total += M.h[I].size();
    }
    M.lmaxDev.alloc(total);
    M.lmaxHost.assign(total, 0.f);
    M.setupVals = nullptr;
    M.built = true;
}

// ---- device: per-tangent set-up -----------------------------------------------------------------------------------
// Galerkin coarse values A_c += P^T A P, one warp per finer node a. First the node's rows of A P: the coarse nodes that
// a's neighbours interpolate from are all neighbours of a's first coarse node i0, so the products are summed in shared
// memory at their rank in i0's list: 4 neighbours at a time (a lane per neighbour and weight looks up the rank), then 8
// weights x 4 lanes of one neighbour add their share of its ncomp^2 values. Then each coarse node i of a takes the rows
// times its weight by atomics. On a lattice a finer node has 43 pairs (i, j) on average, 1.6 times the atomics of its 27
// neighbours alone.
template <typename TA>
__global__ void __launch_bounds__(kBS) k_amg_coarsen(NodeSpmv F, const uint8_t* __restrict__ fmask,
                                                      const TA* __restrict__ fv, NodeSpmv C, int maxList,
                                                      const int32_t* __restrict__ pNode,
                                                      const float* __restrict__ pWeight, TA* cv)
{
    extern __shared__ __align__(16) unsigned char coSmem[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int64_t a = blockIdx.x * static_cast<int64_t>(warps) + wid;
    if (a >= F.totalWarps)
        return;
    const int nc = F.ncomp[0], nc2 = nc * nc;
    TA* acc = reinterpret_cast<TA*>(coSmem) + wid * maxList * nc2;
    int32_t* list = reinterpret_cast<int32_t*>(reinterpret_cast<TA*>(coSmem) + warps * maxList * nc2) + wid * maxList * 2;
    int32_t* rank = list + maxList;
    const int64_t g0 = F.gdof[0][a];
    const int64_t q0 = F.nbrPtr[0][a];
    const int nn = static_cast<int>(F.nbrPtr[0][a + 1] - q0);
    const int32_t i0 = pNode[a * kInterp];
    const int64_t l0 = C.nbrPtr[0][NG_IDX(i0, C.nNodes[0], 31)];
    const int len = static_cast<int>(C.nbrPtr[0][i0 + 1] - l0);
    for (int s = lane; s < len; s += 32)
        list[s] = C.nbrIdx[0][NG_IDX(l0 + s, C.nbrTotal[0], 36)];
    for (int s = lane; s < len * nc2; s += 32)
        acc[s] = TA(0);
    // this lane's values of a neighbour's block: entries sub, sub + 4, sub + 8 of (row c, column d)
    const int sub = lane & 3;
    int64_t row[3];
    int dcol[3];
#pragma unroll
    for (int t = 0; t < 3; ++t)
    {
        const int q = sub + 4 * t, cc = q / nc;
        dcol[t] = q - cc * nc;
        row[t] = q < nc2 && !fmask[g0 + cc] ? F.rowPtr[g0 + cc] + F.blk[0][a] + dcol[t] : -1;
    }
    __syncwarp();
    for (int k0 = 0; k0 < nn; k0 += 4)
    {
        TA v[4][3];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int t = 0; t < 3; ++t)
                v[kk][t] = row[t] >= 0 && k0 + kk < nn ? fv[NG_IDX(row[t] + nc * (k0 + kk), F.nnz, 37)] : TA(0);
        // lane = neighbour (lane / 8) and weight (lane % 8)
        const int k = k0 + (lane >> 3);
        int slot = -1, fixed = 0;
        float w = 0.f;
        if (k < nn)
        {
            const int64_t b = F.nbrIdx[0][NG_IDX(q0 + k, F.nbrTotal[0], 38)];
            const int64_t gb = F.gdof[0][b];
            const int32_t j = pNode[b * kInterp + (lane & 7)];
            w = pWeight[b * kInterp + (lane & 7)];
            for (int d = 0; d < nc; ++d)
                fixed |= (fmask[gb + d] ? 1 : 0) << d;
            if (j >= 0)
            {
                int lo = 0, hi = len - 1; // j is in the list
                while (lo < hi)
                {
                    const int mid = (lo + hi) >> 1;
                    if (list[mid] < j)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                slot = list[lo] == j ? lo : -1;
            }
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
        {
            const int from = kk * 8 + (lane >> 2);
            const int s = __shfl_sync(0xffffffffu, slot, from);
            const int fx = __shfl_sync(0xffffffffu, fixed, from);
            const TA wb = static_cast<TA>(__shfl_sync(0xffffffffu, w, from));
            if (s >= 0)
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    if (row[t] >= 0 && !(fx >> dcol[t] & 1))
                        acc[NG_IDX(s * nc2 + sub + 4 * t, maxList * nc2, 30)] += wb * v[kk][t];
            __syncwarp();
        }
    }
    for (int e = 0; e < kInterp; ++e)
    {
        const int32_t i = pNode[a * kInterp + e];
        if (i < 0)
            break;
        const TA wi = static_cast<TA>(pWeight[a * kInterp + e]);
        const int64_t li = C.nbrPtr[0][NG_IDX(i, C.nNodes[0], 31)];
        const int n = static_cast<int>(C.nbrPtr[0][i + 1] - li);
        for (int s = lane; s < len; s += 32)
        {
            int lo = s;
            if (i != i0)
            {
                const int32_t j = list[s];
                lo = 0;
                int hi = n - 1;
                while (lo < hi)
                {
                    const int mid = (lo + hi) >> 1;
                    if (C.nbrIdx[0][li + mid] < j)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                if (C.nbrIdx[0][li + lo] != j)
                    lo = -1; // no neighbour of a interpolates from it
            }
            rank[s] = lo;
        }
        __syncwarp();
        const int64_t G0 = C.gdof[0][i];
        for (int u = lane; u < len * nc2; u += 32)
        {
            const int s = u / nc2, q = u - s * nc2, cc = q / nc;
            const TA val = wi * acc[u];
            if (rank[s] >= 0 && val != TA(0))
                atomicAdd(cv + NG_IDX(C.rowPtr[G0 + cc] + nc * rank[s] + q - cc * nc, C.nnz, 30), val);
        }
        __syncwarp();
    }
}

// Jacobi diagonal (0 where the DOF is constrained or the diagonal is not positive) and the Gershgorin bound
// max_r sum_j |a_rj| / a_rr of the spectral radius of D^-1 A (positive floats order like their bit patterns)
template <typename TA>
__global__ void __launch_bounds__(kBS) k_amg_diag(NodeSpmv A, const uint8_t* __restrict__ mask,
                                                   const TA* __restrict__ v, const int32_t* __restrict__ diagOff,
                                                   TA* dinv, float* lmax)
{
    const int64_t a = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (a >= A.totalWarps)
        return;
    const int nc = A.ncomp[0];
    const int64_t g0 = A.gdof[0][a];
    const int len = nc * static_cast<int>(A.nbrPtr[0][a + 1] - A.nbrPtr[0][a]);
    for (int c = 0; c < nc; ++c)
    {
        const int64_t r = g0 + c;
        const int64_t rs = A.rowPtr[r] + A.blk[0][a];
        float s = 0.f;
        for (int q = lane; q < len; q += 32)
            s += fabsf(static_cast<float>(v[NG_IDX(rs + q, A.nnz, 32)]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0)
        {
            const TA dg = v[NG_IDX(rs + diagOff[a] + c, A.nnz, 35)];
            const bool use = !mask[r] && dg > TA(0);
            dinv[r] = use ? TA(1) / dg : TA(0);
            if (use)
                atomicMax(reinterpret_cast<int*>(lmax), __float_as_int(s / static_cast<float>(dg)));
        }
    }
}

// ---- device: cycle kernels (each returns at once when the Krylov state is no longer RUN) ------------------------
__device__ __forceinline__ bool Idle(const int* st)
{
    return st && st[ST_STATE] != RUN;
}

// the interpolation entries of node a
template <typename TA>
__device__ __forceinline__ void LoadInterp(const int32_t* __restrict__ pNode, const TA* __restrict__ pWeight, int64_t a,
                                           int32_t (&node)[kInterp], TA (&w)[kInterp])
{
#pragma unroll
    for (int k = 0; k < kInterp; k += 4)
    {
        const int4 n = *reinterpret_cast<const int4*>(pNode + a * kInterp + k);
        node[k] = n.x;
        node[k + 1] = n.y;
        node[k + 2] = n.z;
        node[k + 3] = n.w;
        TA v[4];
        Load4(pWeight + a * kInterp + k, v);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            w[k + q] = v[q];
    }
}

// first Chebyshev step from zero: e = dinv b / theta
template <typename TA>
__global__ void k_cheb0(int64_t n, const TA* __restrict__ dinv, const TA* __restrict__ b, TA* e, TA invTheta, const int* st)
{
    PdlWait();
    PdlTrigger();
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i >= n || Idle(st))
        return;
    e[i] = dinv[i] * b[i] * invTheta;
}

// One product of the cycle with what precedes and follows it, on the padded layout of one slot pair (rows of ncRow
// components, columns of ncCol; the structure of k_spmv_nb: G lanes per node, x of the neighbours gathered into shared
// memory, values streamed with 16-byte loads). With t = A x:
//   GATHER  how x is formed: CG_VECTOR x = xin; CG_ZERO x = dinv b w0 (the first Chebyshev step from zero); CG_PROLONG
//           x = xin + P ce (the coarse correction of unconstrained DOFs)
//   EPI     CE_RESTRICT  cb += P^T (b - t) over unconstrained rows (cb is zero before; with CG_ZERO also xout = x)
//           CE_FIRST     d = dinv (b - t) w1; xout = x + d       (first Chebyshev step from a nonzero x)
//           CE_STEP      d = w2 d + w1 dinv (b - t); xout = x + d (later steps; with CG_ZERO the step before is x itself)
//           CE_RESIDUAL  xout = b - t (constrained rows: b)
// xin and xout differ (other rows still gather xin). At the sizes of the coarse levels a launch is what costs: a level takes
// 3 products. CG_ZERO puts two more loads behind every neighbour of a product that waits for exactly those, CG_PROLONG up to 8
// coarse values per component; on larger levels both run as kernels of their own (kFuseNodes, kProlongNodes). Solves to 1e-13
// with the step from zero in the product on no level / up to 40,000 nodes / on every level: FP32 16^3 11.2 / 10.8 / 10.7 ms,
// 24^3 12.6 / 12.0 / 11.9, 40^3 (68,921 nodes) 25.1 / 24.4 / 24.2; FP64 16^3 11.9 / 11.7 / 11.7, 32^3 (35,937) 34.8 / 35.1 / 35.1,
// 40^3 52.5 / 52.5 / 53.4. The line lies where FP64 stops gaining.
enum CycleGather
{
    CG_VECTOR,
    CG_ZERO,
    CG_PROLONG
};
enum CycleEpilogue
{
    CE_RESTRICT,
    CE_FIRST,
    CE_STEP,
    CE_RESIDUAL
};
constexpr int64_t kFuseNodes = 40000;
constexpr int64_t kProlongNodes = 2500;

// Quadruples of values per row that a lane holds before it has x. FP64: a whole row of 27 neighbours x 3 components, with the
// registers of 2 blocks per SM (20^3: 16.4 us with one quadruple and 3 blocks, 10.9 us); FP32: one, with those of 5 (two to
// three and 4 blocks were 5 % slower at 64^3).
template <typename TA, int G>
constexpr int CycleAhead()
{
    return sizeof(TA) == 4 || G >= 32 ? 1 : (G >= 16 ? 2 : 3);
}
template <typename TA>
constexpr int CycleMinBlocks()
{
    return sizeof(TA) == 4 ? 5 : 2;
}

template <typename TA>
struct CycleArgs
{
    int64_t nNodes, nRows, nbrTotal, nCoarse; // nRows, nbrTotal, nCoarse: extents for checked builds
    int ncRow, ncCol, seg4;
    bool early; // the values may be read before the kernel in front has finished
    const int64_t *gdof, *nbrPtr, *nbBase;
    const int32_t *nbrIdx, *nbrCol, *pNode;
    const TA* pWeight;
    const TA* vals;      // the pair's first padded value
    const uint8_t* mask; // nullptr: no constrained rows
    const TA *b, *dinv, *xin, *ce;
    TA *xout, *d, *cb;
    TA w0, w1, w2;
};

template <typename TA, int G, int GATHER, int EPI>
__global__ void __launch_bounds__(kBS, CycleMinBlocks<TA>()) k_cycle(CycleArgs<TA> A, const int* st)
{
    extern __shared__ __align__(16) unsigned char cySmem[];
    // the structure, and on coarse levels the values, were complete before the kernel in front of this one started: they are
    // fetched while that kernel runs
    const int gl = threadIdx.x & (G - 1);
    TA* xs = reinterpret_cast<TA*>(cySmem) + (threadIdx.x / G) * A.seg4;
    const int64_t a = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / G;
    const bool valid = a < A.nNodes;
    const int ncR = valid ? A.ncRow : 0, ncC = A.ncCol;
    int64_t q0 = 0, g0 = 0;
    int nn = 0;
    const TA* vp = A.vals;
    if (valid)
    {
        q0 = A.nbrPtr[a];
        nn = static_cast<int>(A.nbrPtr[a + 1] - q0);
        vp += A.nbBase[a];
        g0 = A.gdof[a];
    }
    const int sg = (ncC * nn + 3) & ~3;
    int32_t cols[kNbCols];
#pragma unroll
    for (int k = 0; k < kNbCols; ++k)
        cols[k] = gl + k * G < nn ? A.nbrCol[NG_IDX(q0 + gl + k * G, A.nbrTotal, 60)] : 0;
    constexpr int kAhead = CycleAhead<TA, G>();
    TA v0[kAhead][kMaxComp][4];
    auto first = [&]() {
#pragma unroll
        for (int h = 0; h < kAhead; ++h)
#pragma unroll
            for (int c = 0; c < kMaxComp; ++c)
            {
                const int f = 4 * (gl + h * G);
                if (c < ncR && f < sg)
                    Load4(vp + c * sg + f, v0[h][c]);
                else
                    v0[h][c][0] = v0[h][c][1] = v0[h][c][2] = v0[h][c][3] = TA(0);
            }
    };
    if (A.early)
        first();
    PdlWait();
    if (Idle(st))
        return;
    if (!A.early)
        first();
    // x of component c at row g of level node b
    auto value = [&](int64_t g, int64_t b, int c) -> TA {
        if (GATHER == CG_ZERO)
            return A.dinv[g] * A.b[g] * A.w0;
        TA v = A.xin[g];
        if (GATHER == CG_PROLONG && !(A.mask && A.mask[g]))
        {
            int32_t node[kInterp];
            TA w[kInterp];
            LoadInterp(A.pNode, A.pWeight, b, node, w);
#pragma unroll
            for (int k = 0; k < kInterp; ++k)
                if (node[k] >= 0)
                    v += w[k] * A.ce[NG_IDX(static_cast<int64_t>(node[k]) * ncC + c, A.nCoarse, 34)];
        }
        return v;
    };
    auto gather = [&](int t, int64_t col) {
        const int64_t b = GATHER == CG_PROLONG ? A.nbrIdx[q0 + t] : 0;
        for (int d = 0; d < ncC; ++d)
            xs[t * ncC + d] = value(NG_IDX(col + d, A.nRows, 62), b, d);
    };
#pragma unroll
    for (int k = 0; k < kNbCols; ++k)
        if (gl + k * G < nn)
            gather(gl + k * G, cols[k]);
    for (int t = gl + kNbCols * G; t < nn; t += G)
        gather(t, A.nbrCol[NG_IDX(q0 + t, A.nbrTotal, 60)]);
    for (int t = ncC * nn + gl; t < sg; t += G)
        xs[t] = TA(0);
    __syncwarp();
    TA s[kMaxComp];
#pragma unroll
    for (int c = 0; c < kMaxComp; ++c)
        s[c] = TA(0);
#pragma unroll
    for (int h = 0; h < kAhead; ++h)
        if (4 * (gl + h * G) < sg)
        {
            TA xv[4];
            Load4(xs + 4 * (gl + h * G), xv);
#pragma unroll
            for (int c = 0; c < kMaxComp; ++c)
                s[c] += v0[h][c][0] * xv[0] + v0[h][c][1] * xv[1] + v0[h][c][2] * xv[2] + v0[h][c][3] * xv[3];
        }
#pragma unroll 2
    for (int f = 4 * (gl + kAhead * G); f < sg; f += 4 * G)
    {
        TA xv[4];
        Load4(xs + f, xv);
#pragma unroll
        for (int c = 0; c < kMaxComp; ++c)
            if (c < ncR)
            {
                TA v[4];
                Load4(vp + c * sg + f, v);
                s[c] += v[0] * xv[0] + v[1] * xv[1] + v[2] * xv[2] + v[3] * xv[3];
            }
    }
    PdlTrigger();
    int comp;
    const TA t = GroupSum3<G>(s, gl, A.ncRow == 1, comp);
    if (comp < 0 || comp >= ncR)
        return;
    const int64_t r = NG_IDX(g0 + comp, A.nRows, 64);
    const bool fixed = A.mask && A.mask[r];
    if (EPI == CE_RESIDUAL)
    {
        A.xout[r] = fixed ? A.b[r] : A.b[r] - t;
        return;
    }
    const TA x = value(r, a, comp);
    const TA res = A.b[r] - (fixed ? x : t);
    if (EPI == CE_RESTRICT)
    {
        if (GATHER == CG_ZERO)
            A.xout[r] = x;
        if (fixed)
            return;
        int32_t node[kInterp];
        TA w[kInterp];
        LoadInterp(A.pNode, A.pWeight, a, node, w);
#pragma unroll
        for (int k = 0; k < kInterp; ++k)
            if (node[k] >= 0)
                atomicAdd(A.cb + NG_IDX(static_cast<int64_t>(node[k]) * A.ncRow + comp, A.nCoarse, 33),
                          w[k] * res);
        return;
    }
    const TA d = EPI == CE_FIRST ? A.dinv[r] * res * A.w1
                                 : A.w2 * (GATHER == CG_ZERO ? x : A.d[r]) + A.w1 * A.dinv[r] * res;
    A.d[r] = d;
    A.xout[r] = x + d;
}

// Lanes per node and threads per block: 8 lanes (4 for one-component rows and columns, one short segment per node) and 256
// threads stream a large level; on small ones the chain of one node is what takes the time, so more lanes share it and the
// blocks shrink until every SM has one.
template <typename TA, int GATHER, int EPI>
static void LaunchCycle(Ctx& c, const CycleArgs<TA>& A, const int* st)
{
    const bool narrow = A.ncRow == 1 && A.ncCol == 1;
    const int64_t sms = std::max(c.smCount, 1);
    int G = narrow ? 4 : 8;
    const int most = narrow ? 8 : 32;
    while (G < most && A.nNodes * G * 2 <= sms * 512)
        G *= 2;
    const size_t perGroup = static_cast<size_t>(A.seg4) * sizeof(TA);
    int threads = static_cast<int>(std::min<int64_t>(kBS, std::max<int64_t>(32, A.nNodes * G / sms / 32 * 32)));
    while (threads > 32 && (threads / G) * perGroup > 48 * 1024)
        threads -= 32;
    const unsigned blocks = static_cast<unsigned>((A.nNodes * G + threads - 1) / threads);
    const size_t smem = (threads / G) * perGroup;
    if (G == 4)
        NG_CUDA(LaunchPdl(k_cycle<TA, 4, GATHER, EPI>, blocks, threads, smem, c.stream, A, st));
    else if (G == 8)
        NG_CUDA(LaunchPdl(k_cycle<TA, 8, GATHER, EPI>, blocks, threads, smem, c.stream, A, st));
    else if (G == 16)
        NG_CUDA(LaunchPdl(k_cycle<TA, 16, GATHER, EPI>, blocks, threads, smem, c.stream, A, st));
    else
        NG_CUDA(LaunchPdl(k_cycle<TA, 32, GATHER, EPI>, blocks, threads, smem, c.stream, A, st));
    c.stats.kernel_launches += 1;
}

// e += P ce on the unconstrained rows, one thread per row
template <typename TA>
__global__ void k_prolong(NodeSpmv F, const uint8_t* __restrict__ fmask, const int32_t* __restrict__ pNode,
                          const TA* __restrict__ pWeight, int64_t nCoarse, const TA* __restrict__ ce, TA* e,
                          const int* st)
{
    PdlWait();
    PdlTrigger();
    const int nc = F.ncomp[0];
    const int64_t u = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x, a = u / nc;
    if (a >= F.totalWarps || Idle(st))
        return;
    const int c = static_cast<int>(u - a * nc);
    const int64_t r = F.gdof[0][a] + c;
    if (fmask[r])
        return;
    int32_t node[kInterp];
    TA w[kInterp];
    LoadInterp(pNode, pWeight, a, node, w);
    TA s = e[r];
#pragma unroll
    for (int k = 0; k < kInterp; ++k)
        if (node[k] >= 0)
            s += w[k] * ce[NG_IDX(static_cast<int64_t>(node[k]) * nc + c, nCoarse, 34)];
    e[r] = s;
}

template <typename TA, typename TB>
__global__ void k_convert(int64_t n, const TA* __restrict__ a, TB* __restrict__ b, const int* st)
{
    PdlWait();
    PdlTrigger();
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n && !Idle(st))
        b[i] = static_cast<TB>(a[i]);
}

// ---- device: the coarsest levels in one block ----------------------------------------------------------------
// Levels with at most kTailNodes nodes (and every coarser one) do microseconds of work per launch. Their whole V-cycle is a
// fixed linear map of at most 384 values, so it is formed once per tangent as a dense matrix: block k of k_amg_tail runs the
// cycle on unit vector k (the same Chebyshev recurrences, coefficients from the same double-precision formulas, the same
// restriction and prolongation, a warp-per-node product on the coarse node-block CSR, block barriers between the steps),
// and every sweep applies it with one small product. Run once per sweep in one block instead, the cycle took 55-73 us per
// slot in FP32 and more in FP64, whose pipe is 2 lanes per clock and SM; the product takes 3-6 us, forming the matrix (90 nodes
// x 3) 150 us in FP32 and 227 us in FP64 per tangent. Solves to 1e-13 with the fused cycle (k_cycle) and this: FP32 24^3
// 130 -> 69 ms, FP64 20^3 203 -> 123 ms (launches per iteration 92 -> 33).
constexpr int kTailNodes = 128;
constexpr int kTailMax = 8;
constexpr int kTailThreads = 1024;

template <typename TA>
struct TailLevel
{
    const int64_t* rowPtr;
    const int64_t* nbrPtr;
    const int32_t* nbrCol;
    const int32_t* pNode; // interpolation from the next coarser level (unused on the coarsest)
    const TA* pWeight;
    const TA* vals;
    const TA* dinv;
    TA *b, *e, *t, *d;
    int64_t nNodes, nnz, nDofs, nbrTotal;
    int ncomp;
    double lmax;
};

template <typename TA>
struct TailArgs
{
    int nl;
    int pre, post, coarse;
    double smoothRatio, coarseRatio;
    TailLevel<TA> L[kTailMax];
    int64_t stride; // block k works on vectors k * stride behind the levels'
    TA* columns;    // [k][i]: block k's result
};

template <typename TA>
__device__ void TailSpmv(const TailLevel<TA>& L, const TA* __restrict__ x, TA* __restrict__ y)
{
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int nc = L.ncomp;
    for (int64_t a = threadIdx.x >> 5; a < L.nNodes; a += nw)
    {
        const int64_t q0 = L.nbrPtr[a];
        const int len = static_cast<int>(L.nbrPtr[a + 1] - q0) * nc;
        TA s[kMaxComp];
#pragma unroll
        for (int c = 0; c < kMaxComp; ++c)
            s[c] = TA(0);
        for (int q = lane; q < len; q += 32)
        {
            const int k = q / nc, d = q - k * nc;
            const TA xv = x[NG_IDX(L.nbrCol[NG_IDX(q0 + k, L.nbrTotal, 70)] + d, L.nDofs, 71)];
#pragma unroll
            for (int c = 0; c < kMaxComp; ++c)
                if (c < nc)
                    s[c] += L.vals[NG_IDX(L.rowPtr[a * nc + c] + q, L.nnz, 72)] * xv;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < kMaxComp; ++c)
                s[c] += __shfl_down_sync(0xffffffffu, s[c], o);
        if (lane == 0)
            for (int c = 0; c < nc; ++c)
                y[a * nc + c] = s[c];
    }
}

// Chebyshev smoothing of A e = b on [lmax / ratio, lmax]; ends with a block barrier
template <typename TA>
__device__ void TailCheb(const TailLevel<TA>& L, int degree, bool fromZero, double ratio)
{
    const double lmax = L.lmax, lmin = L.lmax / ratio;
    const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
    const double sigma = theta / delta;
    double rho = 1. / sigma;
    const TA invTheta = TA(1. / theta);
    if (fromZero)
    {
        for (int64_t i = threadIdx.x; i < L.nDofs; i += blockDim.x)
        {
            const TA v = L.dinv[i] * L.b[i] * invTheta;
            L.d[i] = v;
            L.e[i] = v;
        }
    }
    else
    {
        TailSpmv(L, L.e, L.t);
        __syncthreads();
        for (int64_t i = threadIdx.x; i < L.nDofs; i += blockDim.x)
        {
            const TA v = L.dinv[i] * (L.b[i] - L.t[i]) * invTheta;
            L.d[i] = v;
            L.e[i] += v;
        }
    }
    __syncthreads();
    for (int k = 1; k < degree; ++k)
    {
        const double rhoNew = 1. / (2. * sigma - rho);
        const TA c1 = TA(rhoNew * rho), c2 = TA(2. * rhoNew / delta);
        TailSpmv(L, L.e, L.t);
        __syncthreads();
        for (int64_t i = threadIdx.x; i < L.nDofs; i += blockDim.x)
        {
            const TA v = c1 * L.d[i] + c2 * L.dinv[i] * (L.b[i] - L.t[i]);
            L.d[i] = v;
            L.e[i] += v;
        }
        __syncthreads();
        rho = rhoNew;
    }
}

// Block k runs the V-cycle of the tail levels on unit vector k of the first level and stores the result as column k of the
// tail's matrix (TailDense).
template <typename TA>
__global__ void __launch_bounds__(kTailThreads) k_amg_tail(TailArgs<TA> T)
{
    __shared__ TailLevel<TA> L[kTailMax];
    for (int l = threadIdx.x; l < T.nl; l += blockDim.x)
    {
        TailLevel<TA> F = T.L[l];
        const int64_t o = blockIdx.x * T.stride;
        F.b += o;
        F.e += o;
        F.t += o;
        F.d += o;
        L[l] = F;
    }
    __syncthreads();
    for (int64_t i = threadIdx.x; i < L[0].nDofs; i += blockDim.x)
        L[0].b[i] = i == blockIdx.x ? TA(1) : TA(0);
    __syncthreads();
    for (int l = 0; l + 1 < T.nl; ++l)
    {
        const TailLevel<TA>& F = L[l];
        const TailLevel<TA>& C = L[l + 1];
        TailCheb(F, T.pre, true, T.smoothRatio);
        TailSpmv(F, F.e, F.t);
        for (int64_t i = threadIdx.x; i < C.nDofs; i += blockDim.x)
            C.b[i] = TA(0);
        __syncthreads();
        for (int64_t a = threadIdx.x; a < F.nNodes; a += blockDim.x)
        {
            int32_t node[kInterp];
            TA w[kInterp];
            LoadInterp(F.pNode, F.pWeight, a, node, w);
            for (int c = 0; c < F.ncomp; ++c)
            {
                const TA res = F.b[a * F.ncomp + c] - F.t[a * F.ncomp + c];
#pragma unroll
                for (int k = 0; k < kInterp; ++k)
                    if (node[k] >= 0)
                        atomicAdd(C.b + NG_IDX(static_cast<int64_t>(node[k]) * C.ncomp + c, C.nDofs, 73),
                                  w[k] * res);
            }
        }
        __syncthreads();
    }
    TailCheb(L[T.nl - 1], T.coarse, true, T.coarseRatio);
    for (int l = T.nl - 2; l >= 0; --l)
    {
        const TailLevel<TA>& F = L[l];
        const TailLevel<TA>& C = L[l + 1];
        for (int64_t a = threadIdx.x; a < F.nNodes; a += blockDim.x)
        {
            int32_t node[kInterp];
            TA w[kInterp];
            LoadInterp(F.pNode, F.pWeight, a, node, w);
            for (int c = 0; c < F.ncomp; ++c)
            {
                TA s = F.e[a * F.ncomp + c];
#pragma unroll
                for (int k = 0; k < kInterp; ++k)
                    if (node[k] >= 0)
                        s += w[k] * C.e[NG_IDX(static_cast<int64_t>(node[k]) * C.ncomp + c, C.nDofs, 74)];
                F.e[a * F.ncomp + c] = s;
            }
        }
        __syncthreads();
        TailCheb(F, T.post, false, T.smoothRatio);
    }
    const int64_t n = L[0].nDofs;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
        T.columns[blockIdx.x * n + i] = L[0].e[i];
}

// e = M b with the tail's matrix (columns m[k]): a block owns 32 rows, its warps a share of the columns each
constexpr int kDenseWarps = 16;
template <typename TA>
__global__ void __launch_bounds__(kDenseWarps * 32) k_amg_tail_dense(int n, const TA* __restrict__ m,
                                                                     const TA* __restrict__ b, TA* __restrict__ e,
                                                                     const int* st)
{
    PdlWait();
    PdlTrigger();
    __shared__ TA part[kDenseWarps][32];
    if (Idle(st))
        return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    TA s = TA(0);
    if (i < n)
    {
#pragma unroll 8
        for (int k = wid; k < n; k += kDenseWarps)
            s += m[static_cast<int64_t>(k) * n + i] * b[k];
    }
    part[wid][lane] = s;
    __syncthreads();
    if (wid == 0 && i < n)
    {
        TA t = TA(0);
#pragma unroll
        for (int w = 0; w < kDenseWarps; ++w)
            t += part[w][lane];
        e[i] = t;
    }
}

// ---- host: set-up and application ------------------------------------------------------------------------------
static unsigned Blocks(int64_t n, int bs = 256)
{
    return static_cast<unsigned>((n + bs - 1) / bs);
}

// device vectors of every level in arithmetic TA (on first use of TA)
template <typename TA>
static void EnsureNum(Ctx& c, Amg& M)
{
    int64_t rhs = 0;
    for (int I = 0; I < M.ns; ++I)
        for (size_t l = 0; l < M.h[I].size(); ++l)
        {
            AmgLevel& L = M.h[I][l];
            Num<TA>& U = N<TA>(L);
            const int64_t n = l == 0 ? c.nDofs : L.nDofs;
            rhs += l > 0 ? L.nDofs : 0;
            if (U.dinv.n == static_cast<size_t>(n))
                continue;
            if (l > 0)
            {
                LevelNodes& X = *L.nodes;
                if (sizeof(TA) == 8 && X.pWeight64.n != X.pWeight.n)
                {
                    X.pWeight64.alloc(X.pWeight.n);
                    const int64_t m = static_cast<int64_t>(X.pWeight.n);
                    k_convert<float, double><<<Blocks(m), 256, 0, c.stream>>>(m, X.pWeight.p, X.pWeight64.p, nullptr);
                    c.stats.kernel_launches += 1;
                }
                U.vals.alloc(L.nnz);
                U.nb.alloc(std::max<int64_t>(L.nbTotal, 4));
            }
            for (DBuf<TA>* b : {&U.dinv, &U.e, &U.t, &U.d})
                b->alloc(n);
        }
    DBuf<TA>& R = Rhs<TA>(M);
    if (R.n != static_cast<size_t>(rhs))
    {
        R.alloc(rhs);
        int64_t at = 0;
        for (int I = 0; I < M.ns; ++I)
            for (size_t l = 1; l < M.h[I].size(); ++l)
            {
                N<TA>(M.h[I][l]).b = R.p + at;
                at += M.h[I][l].nDofs;
            }
    }
}

// first level (>= 1) from which every level has at most kTailNodes nodes, if they fit one tail launch; 0: none
static size_t TailStart(const std::vector<AmgLevel>& H)
{
    for (size_t l = 1; l < H.size(); ++l)
        if (H[l].nNodes <= kTailNodes)
            return H.size() - l <= static_cast<size_t>(kTailMax) ? l : 0;
    return 0;
}

// the dense matrix of slot I's tail for the current coarse operators
template <typename TA>
static void BuildTail(Ctx& c, int I, bool sym)
{
    Amg& M = *c.amg;
    std::vector<AmgLevel>& H = M.h[I];
    const size_t l0 = TailStart(H);
    TailDense<TA>& D = Tail<TA>(M, I);
    if (l0 == 0)
    {
        D.n = 0;
        return;
    }
    int64_t sum = 0; // values of one level-vector set
    for (size_t l = l0; l < H.size(); ++l)
        sum += H[l].nDofs;
    D.n = H[l0].nDofs;
    if (D.m.n != static_cast<size_t>(D.n * D.n))
        D.m.alloc(D.n * D.n);
    if (D.work.n != static_cast<size_t>(4 * sum * D.n))
        D.work.alloc(4 * sum * D.n);
    TailArgs<TA> T{};
    T.nl = static_cast<int>(H.size() - l0);
    T.pre = sym ? kPostDegree : kPreDegree;
    T.post = kPostDegree;
    T.coarse = CoarseDegree<TA>();
    T.smoothRatio = kSmoothRatio;
    T.coarseRatio = kCoarseRatio;
    T.stride = 4 * sum;
    T.columns = D.m.p;
    int64_t at = 0;
    for (int k = 0; k < T.nl; ++k)
    {
        AmgLevel& Lk = H[l0 + k];
        Num<TA>& Uk = N<TA>(Lk);
        TailLevel<TA>& F = T.L[k];
        F.rowPtr = Lk.rowPtr.p;
        F.nbrPtr = Lk.nodes->dNbrPtr.p;
        F.nbrCol = Lk.nbrCol.p;
        F.pNode = l0 + k + 1 < H.size() ? H[l0 + k + 1].nodes->pNode.p : nullptr;
        F.pWeight = l0 + k + 1 < H.size() ? Weights<TA>(*H[l0 + k + 1].nodes).p : nullptr;
        F.vals = Uk.vals.p;
        F.dinv = Uk.dinv.p;
        for (TA** v : {&F.b, &F.e, &F.t, &F.d})
        {
            *v = D.work.p + at;
            at += Lk.nDofs;
        }
        F.nNodes = Lk.nNodes;
        F.nnz = Lk.nnz;
        F.nDofs = Lk.nDofs;
        F.nbrTotal = static_cast<int64_t>(Lk.nodes->dNbrIdx.n);
        F.ncomp = Lk.ncomp;
        F.lmax = Lk.lmax;
    }
    k_amg_tail<TA><<<static_cast<unsigned>(D.n), kTailThreads, 0, c.stream>>>(T);
    AfterLaunch(c, "k_amg_tail");
    c.stats.kernel_launches += 1;
}

// Builds the hierarchy on first use and the coarse operators for the tangent `vals` unless they were built for
// the same values already (same pointer and tangent version). The preconditioner works in the arithmetic of the
// tangent values: FP32 for FP32 tangents, FP64 for FP64 tangents.
template <typename TV>
void AmgSetup(Ctx& c, const TV* vals, bool sym)
{
    HostClock hc(&c.hostMs[HP_AMG_SETUP]);
    if (!c.amg)
    {
        c.amg = new Amg();
        const char* gr = std::getenv("NUTO_GPU_GRAPHS");
        c.amg->graphs = !(gr && gr[0] == '0');
    }
    Amg& M = *c.amg;
    if (!M.built)
        BuildHierarchy(c);
    if (M.setupVals == static_cast<const void*>(vals) && M.setupVersion == c.valsVersion)
    {
        if (M.tailSym != sym) // the same values for the other Krylov method: its cycle differs in the pre-smoothing
        {
            for (int I = 0; I < M.ns; ++I)
                BuildTail<TV>(c, I, sym);
            M.tailSym = sym;
        }
        return;
    }
    EnsureNum<TV>(c, M);
    M.prec = sizeof(TV) == 4 ? 32 : 64;
    M.fine = vals;
    NG_CUDA(cudaMemsetAsync(M.lmaxDev.p, 0, M.lmaxHost.size() * sizeof(float), c.stream));
    size_t slot = 0;
    for (int I = 0; I < M.ns; ++I)
    {
        std::vector<AmgLevel>& H = M.h[I];
        H[0].spmv = SlotView(c, I);
        k_amg_diag<TV><<<Blocks(H[0].nNodes * 32), kBS, 0, c.stream>>>(H[0].spmv, c.dMask.p, vals, H[0].diagOff.p,
                                                                        N<TV>(H[0]).dinv.p, M.lmaxDev.p + slot);
        c.stats.kernel_launches += 1;
        for (size_t l = 1; l < H.size(); ++l)
        {
            AmgLevel& Fi = H[l - 1];
            AmgLevel& C = H[l];
            Num<TV>& CU = N<TV>(C);
            NG_CUDA(cudaMemsetAsync(CU.vals.p, 0, C.nnz * sizeof(TV), c.stream));
            const size_t perWarp = C.nodes->maxList * (C.ncomp * C.ncomp * sizeof(TV) + 2 * sizeof(int32_t));
            const int warps = static_cast<int>(std::max<size_t>(1, std::min<size_t>(kBS / 32, 48 * 1024 / perWarp)));
            k_amg_coarsen<TV><<<Blocks(Fi.nNodes, warps), warps * 32, warps * perWarp, c.stream>>>(
                    Fi.spmv, l == 1 ? c.dMask.p : Fi.zeroMask.p, l == 1 ? vals : N<TV>(Fi).vals.p, C.spmv, C.nodes->maxList,
                    C.nodes->pNode.p, C.nodes->pWeight.p, CU.vals.p);
            k_amg_diag<TV><<<Blocks(C.nNodes * 32), kBS, 0, c.stream>>>(C.spmv, C.zeroMask.p, CU.vals.p, C.diagOff.p,
                                                                         CU.dinv.p, M.lmaxDev.p + slot + l);
            c.stats.kernel_launches += 2;
            if (C.nbTotal > 0)
            {
                // the level's products stream the padded layout (filled from the new Galerkin values)
                NodeSpmv& V = C.spmv;
                V.nbBase[0] = C.nbBase.p;
                V.nbOff[0] = 0;
                V.nbSeg4 = C.nbSeg4;
                V.ncMaxRows = C.ncomp;
                if constexpr (sizeof(TV) == 4)
                {
                    V.nb32 = CU.nb.p;
                    V.nbSrc32 = CU.vals.p;
                }
                else
                {
                    V.nb64 = CU.nb.p;
                    V.nbSrc64 = CU.vals.p;
                }
                k_nb_pack<TV><<<Blocks(C.nNodes * 32), kBS, 0, c.stream>>>(V, CU.vals.p, CU.nb.p);
                c.stats.kernel_launches += 1;
            }
        }
        slot += H.size();
    }
    AfterLaunch(c, "multigrid set-up");
    NG_CUDA(cudaMemcpyAsync(M.lmaxHost.data(), M.lmaxDev.p, M.lmaxHost.size() * sizeof(float),
                            cudaMemcpyDeviceToHost, c.stream));
    NG_CUDA(cudaStreamSynchronize(c.stream));
    slot = 0;
    for (int I = 0; I < M.ns; ++I)
        for (AmgLevel& L : M.h[I])
        {
            const float v = M.lmaxHost[slot++];
            L.lmax = v > 0.f ? v : 1.f;
        }
    for (int I = 0; I < M.ns; ++I)
        BuildTail<TV>(c, I, sym);
    M.tailSym = sym;
    M.setupVals = vals;
    M.setupVersion = c.valsVersion;
    M.setups++;
}
template void AmgSetup<float>(Ctx&, const float*, bool);
template void AmgSetup<double>(Ctx&, const double*, bool);

// Chebyshev coefficients on [lmax / ratio, lmax]: step k multiplies the last step by w2 and dinv (b - A e) by w1
struct Cheb
{
    double theta, delta, sigma, rho;
    Cheb(const AmgLevel& L, float ratio)
    {
        const double lmax = L.lmax, lmin = L.lmax / ratio;
        theta = 0.5 * (lmax + lmin);
        delta = 0.5 * (lmax - lmin);
        sigma = theta / delta;
        rho = 1. / sigma;
    }
    void step(double& w2, double& w1)
    {
        const double rhoNew = 1. / (2. * sigma - rho);
        w2 = rhoNew * rho;
        w1 = 2. * rhoNew / delta;
        rho = rhoNew;
    }
};

// the diagonal block of a level for k_cycle (vectors are base pointers of the level: combined length on level 0)
template <typename TA>
static CycleArgs<TA> LevelArgs(Ctx& c, AmgLevel& L, bool fine)
{
    const NodeSpmv& V = L.spmv;
    CycleArgs<TA> A{};
    NG_CHECK(SpmvPadded(V, fine ? static_cast<const TA*>(c.amg->fine) : N<TA>(L).vals.p), NUTO_GPU_ESTATE,
             "the padded layout does not hold the level's values");
    A.nNodes = L.nNodes;
    A.nRows = V.nRows;
    A.nbrTotal = V.nbrTotal[0];
    A.ncRow = A.ncCol = L.ncomp;
    A.seg4 = V.nbSeg4;
    A.gdof = V.gdof[0];
    A.nbrPtr = V.nbrPtr[0];
    A.nbrCol = V.nbrCol[0];
    A.nbrIdx = V.nbrIdx[0];
    A.early = !fine; // filled by the set-up, which ends with a synchronisation
    A.nbBase = V.nbBase[0];
    A.vals = NbValues<TA>(V) + V.nbOff[0];
    A.mask = fine ? c.dMask.p : nullptr;
    A.dinv = N<TA>(L).dinv.p;
    A.d = N<TA>(L).d.p;
    return A;
}

// e = V-cycle(b) on level l of slot I's hierarchy
template <typename TA>
static void VCycle(Ctx& c, int I, size_t l, const TA* b, TA* e, const int* st, bool sym)
{
    Amg& M = *c.amg;
    std::vector<AmgLevel>& H = M.h[I];
    AmgLevel& L = H[l];
    Num<TA>& U = N<TA>(L);
    if (l > 0 && l == TailStart(H))
    {
        const TailDense<TA>& D = Tail<TA>(M, I);
        NG_CUDA(LaunchPdl(k_amg_tail_dense<TA>, Blocks(D.n, 32), kDenseWarps * 32, 0, c.stream, static_cast<int>(D.n), D.m.p,
                          b, e, st));
        c.stats.kernel_launches += 1;
        return;
    }
    CycleArgs<TA> A = LevelArgs<TA>(c, L, l == 0);
    A.b = b;
    const int64_t n = L.nDofs, o = L.off;
    const bool fuse = L.nNodes <= kFuseNodes;
    // from zero: x = dinv b / theta, in the product's gather or in a kernel of its own (into `to`)
    auto fromZero = [&](const Cheb& C, TA* to) {
        A.w0 = TA(1. / C.theta);
        if (fuse)
            return;
        NG_CUDA(LaunchPdl(k_cheb0<TA>, Blocks(n), 256, 0, c.stream, n, U.dinv.p + o, b + o, to + o, A.w0, st));
        c.stats.kernel_launches += 1;
        A.xin = to;
    };
    auto stepFromZero = [&](TA* out) {
        A.xout = out;
        if (fuse)
            LaunchCycle<TA, CG_ZERO, CE_STEP>(c, A, st);
        else
        {
            // the step before is x itself: d = x
            NG_CUDA(cudaMemcpyAsync(U.d.p + o, A.xin + o, n * sizeof(TA), cudaMemcpyDeviceToDevice, c.stream));
            LaunchCycle<TA, CG_VECTOR, CE_STEP>(c, A, st);
        }
    };
    auto coefficients = [&](Cheb& C) {
        double w2, w1;
        C.step(w2, w1);
        A.w1 = TA(w1);
        A.w2 = TA(w2);
    };
    if (l + 1 == H.size())
    {
        // Chebyshev solve; the steps alternate between t and e and end in e
        Cheb C(L, kCoarseRatio);
        const int steps = CoarseDegree<TA>() - 1;
        TA* buf[2] = {U.t.p, e}; // step s writes buf[(steps - s) & 1 ? 0 : 1]
        fromZero(C, steps & 1 ? U.t.p : e);
        for (int s = 1; s <= steps; ++s)
        {
            coefficients(C);
            TA* out = buf[(steps - s) & 1 ? 0 : 1];
            if (s == 1)
                stepFromZero(out);
            else
            {
                A.xout = out;
                LaunchCycle<TA, CG_VECTOR, CE_STEP>(c, A, st);
            }
            A.xin = out;
        }
        return;
    }
    AmgLevel& Co = H[l + 1];
    Num<TA>& CU = N<TA>(Co);
    // pre-smoothing from zero (one step, two in the symmetric cycle), then the residual restricted
    A.pNode = Co.nodes->pNode.p;
    A.pWeight = Weights<TA>(*Co.nodes).p;
    A.cb = CU.b;
    A.nCoarse = Co.nDofs;
    {
        Cheb C(L, kSmoothRatio);
        if (sym)
        {
            fromZero(C, U.t.p);
            coefficients(C);
            stepFromZero(e);
            A.xin = e;
            LaunchCycle<TA, CG_VECTOR, CE_RESTRICT>(c, A, st);
        }
        else
        {
            fromZero(C, e);
            A.xout = e;
            if (fuse)
                LaunchCycle<TA, CG_ZERO, CE_RESTRICT>(c, A, st);
            else
                LaunchCycle<TA, CG_VECTOR, CE_RESTRICT>(c, A, st);
        }
    }
    VCycle<TA>(c, I, l + 1, CU.b, CU.e.p, st, sym);
    // coarse correction and two post-smoothing steps: e -> t -> e
    A.xin = e;
    A.xout = U.t.p;
    A.ce = CU.e.p;
    Cheb C(L, kSmoothRatio);
    A.w1 = TA(1. / C.theta);
    bool prolonged = false;
    if constexpr (sizeof(TA) == 4)
        if (L.nNodes <= kProlongNodes)
        {
            LaunchCycle<TA, CG_PROLONG, CE_FIRST>(c, A, st);
            prolonged = true;
        }
    if (!prolonged)
    {
        NG_CUDA(LaunchPdl(k_prolong<TA>, Blocks(n), 256, 0, c.stream, L.spmv, l == 0 ? c.dMask.p : L.zeroMask.p,
                          static_cast<const int32_t*>(Co.nodes->pNode.p), static_cast<const TA*>(Weights<TA>(*Co.nodes).p),
                          Co.nDofs, static_cast<const TA*>(CU.e.p), e, st));
        c.stats.kernel_launches += 1;
        LaunchCycle<TA, CG_VECTOR, CE_FIRST>(c, A, st);
    }
    static_assert(kPostDegree == 2, "two post-smoothing steps");
    coefficients(C);
    A.xin = U.t.p;
    A.xout = e;
    LaunchCycle<TA, CG_VECTOR, CE_STEP>(c, A, st);
}

// block Gauss-Seidel sweep in slot order on combined vectors: z_0 = V_0(v_0), z_1 = V_1(v_1 - K_10 z_0)
template <typename TA>
static void Sweep(Ctx& c, const TA* v, TA* z, TA* res, const int* st, bool sym)
{
    Amg& M = *c.amg;
    if (Rhs<TA>(M).n > 0)
        NG_CUDA(cudaMemsetAsync(Rhs<TA>(M).p, 0, Rhs<TA>(M).n * sizeof(TA), c.stream));
    VCycle<TA>(c, 0, 0, v, z, st, sym);
    for (int I = 1; I < M.ns; ++I)
    {
        // res = v_I - K_I0 z_0 on the rows of slot I
        const PairMap& P = c.pairs[I * M.ns];
        const NbLayout::Pair& nb = c.nb.pair[I * M.ns];
        CycleArgs<TA> A{};
        A.nNodes = c.slots[I].nNodes;
        A.nRows = c.nDofs;
        A.nbrTotal = static_cast<int64_t>(P.dNbrIdx.n);
        A.ncRow = c.slots[I].ncomp;
        A.ncCol = c.slots[0].ncomp;
        A.seg4 = nb.maxSeg4;
        A.gdof = c.slots[I].dGdof.p;
        A.nbrPtr = P.dNbrPtr.p;
        A.nbrCol = P.dNbrCol.p;
        A.nbBase = nb.base.p;
        A.vals = NbValues<TA>(M.h[I][0].spmv) + nb.off;
        A.mask = c.dMask.p;
        A.b = v;
        A.xin = z;
        A.xout = res;
        LaunchCycle<TA, CG_VECTOR, CE_RESIDUAL>(c, A, st);
        VCycle<TA>(c, I, 0, res, z, st, sym);
    }
}

// Runs Sweep<TA>(in, out) through the graph of (TA, sym), capturing or updating it when the set-up changed. Returns
// false when graphs are off or the capture failed (the caller then launches the sweep kernel by kernel).
template <typename TA>
static bool SweepGraphRun(Ctx& c, TA* in, TA* out, TA* res, const int* st, bool sym)
{
    Amg& M = *c.amg;
    if (!M.graphs)
        return false;
    SweepGraph& G = M.graph[sizeof(TA) == 8 ? 1 : 0][sym ? 1 : 0];
    if (!G.exec || G.setup != M.setups || G.st != st)
    {
        HostClock hc(&c.hostMs[HP_GRAPH]);
        const int64_t before = c.stats.kernel_launches;
        cudaGraph_t graph = nullptr;
        // Capture on a private stream: capture is not permitted on the legacy default stream, which a caller may
        // hand to nuto_gpu_create. Capturing records the launches without running them, so swapping the
        // context's stream for the duration does not reorder any work; the graph is launched on the context's
        // stream.
        if (!M.capStream)
            NG_CUDA(cudaStreamCreateWithFlags(&M.capStream, cudaStreamNonBlocking));
        const cudaError_t eb = cudaStreamBeginCapture(M.capStream, cudaStreamCaptureModeThreadLocal);
        if (eb != cudaSuccess)
        {
            cudaGetLastError();
            M.graphs = false;
            M.graphError = std::string("begin capture: ") + cudaGetErrorString(eb);
            return false;
        }
        const cudaStream_t own = c.stream;
        c.stream = M.capStream;
        try
        {
            Sweep<TA>(c, in, out, res, st, sym);
        }
        catch (...)
        {
            c.stream = own;
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(M.capStream, &g);
            if (g)
                cudaGraphDestroy(g);
            cudaGetLastError();
            throw;
        }
        c.stream = own;
        const cudaError_t ec = cudaStreamEndCapture(M.capStream, &graph);
        G.launches = c.stats.kernel_launches - before;
        c.stats.kernel_launches = before;
        bool ok = ec == cudaSuccess && graph != nullptr;
        if (!ok)
            M.graphError = std::string("end capture: ") + cudaGetErrorString(ec);
        if (ok && G.exec)
        {
            cudaGraphExecUpdateResultInfo info;
            if (cudaGraphExecUpdate(G.exec, graph, &info) != cudaSuccess)
            {
                cudaGetLastError();
                cudaGraphExecDestroy(G.exec);
                G.exec = nullptr;
            }
        }
        if (ok && !G.exec)
        {
            const cudaError_t ei = cudaGraphInstantiate(&G.exec, graph, 0);
            ok = ei == cudaSuccess;
            if (!ok)
                M.graphError = std::string("instantiate: ") + cudaGetErrorString(ei);
        }
        if (graph)
            cudaGraphDestroy(graph);
        if (!ok)
        {
            cudaGetLastError();
            if (G.exec)
                cudaGraphExecDestroy(G.exec);
            G.exec = nullptr;
            M.graphs = false;
            return false;
        }
        G.setup = M.setups;
        G.st = st;
    }
    NG_CUDA(cudaGraphLaunch(G.exec, c.stream));
    M.graphLaunched = true;
    c.stats.kernel_launches += G.launches;
    return true;
}

template <typename T>
void AmgVectors(Ctx& c, T** in, T** out)
{
    Amg& M = *c.amg;
    *in = *out = nullptr;
    if (M.prec != static_cast<int>(8 * sizeof(T)))
        return;
    DBuf<T>*vi, *vo, *vr;
    if constexpr (sizeof(T) == 4)
    {
        vi = &M.in32;
        vo = &M.out32;
        vr = &M.res32;
    }
    else
    {
        vi = &M.in64;
        vo = &M.out64;
        vr = &M.res64;
    }
    for (DBuf<T>* b : {vi, vo, vr})
        if (b->n != static_cast<size_t>(c.nDofs))
            b->alloc(c.nDofs);
    *in = vi->p;
    *out = vo->p;
}
template void AmgVectors<float>(Ctx&, float**, float**);
template void AmgVectors<double>(Ctx&, double**, double**);

template <typename T>
void AmgSweep(Ctx& c, const int* st, bool sym)
{
    T *in, *out, *res;
    AmgVectors<T>(c, &in, &out);
    if constexpr (sizeof(T) == 4)
        res = c.amg->res32.p;
    else
        res = c.amg->res64.p;
    if (!SweepGraphRun<T>(c, in, out, res, st, sym))
        Sweep<T>(c, in, out, res, st, sym);
}
template void AmgSweep<float>(Ctx&, const int*, bool);
template void AmgSweep<double>(Ctx&, const int*, bool);

// z = M^-1 v for the tangent of the last AmgSetup, in that tangent's arithmetic (FP64 Krylov vectors with an
// FP32 tangent are converted). With st given, every kernel returns at once when the Krylov state is not RUN.
// sym = true runs equal pre- and post-smoothing (a symmetric cycle for PCG on a single slot); otherwise the
// cheaper V(1,2) for GMRES. The sweep runs as a CUDA graph on fixed vectors (input and output copied).
template <typename T>
void AmgApply(Ctx& c, const T* v, T* z, const int* st, bool sym)
{
    const int64_t n = c.nDofs;
    T *in, *out;
    AmgVectors<T>(c, &in, &out);
    if (in)
    {
        NG_CUDA(cudaMemcpyAsync(in, v, n * sizeof(T), cudaMemcpyDeviceToDevice, c.stream));
        AmgSweep<T>(c, st, sym);
        NG_CUDA(cudaMemcpyAsync(z, out, n * sizeof(T), cudaMemcpyDeviceToDevice, c.stream));
        return;
    }
    if constexpr (sizeof(T) == 8)
    {
        float *in32, *out32;
        AmgVectors<float>(c, &in32, &out32);
        NG_CUDA(LaunchPdl(k_convert<double, float>, Blocks(n), 256, 0, c.stream, n, v, in32, st));
        AmgSweep<float>(c, st, sym);
        NG_CUDA(LaunchPdl(k_convert<float, double>, Blocks(n), 256, 0, c.stream, n, static_cast<const float*>(out32), z, st));
        c.stats.kernel_launches += 2;
    }
    else
        throw Error{NUTO_GPU_EINVAL, "FP32 Krylov vectors with an FP64 multigrid set-up"};
}
template void AmgApply<float>(Ctx&, const float*, float*, const int*, bool);
template void AmgApply<double>(Ctx&, const double*, double*, const int*, bool);

bool AmgGraphActive(const Ctx& c)
{
    return c.amg && c.amg->graphs && c.amg->graphLaunched;
}

const char* AmgGraphStatus(const Ctx& c)
{
    if (!c.amg)
        return "no multigrid";
    if (c.amg->graphs)
        return "sweep graph on";
    return c.amg->graphError.empty() ? "sweep graph off" : c.amg->graphError.c_str();
}

int AmgLevels(const Ctx& c)
{
    return c.amg ? static_cast<int>(c.amg->h[0].size()) : 0;
}

} // namespace nuto_gpu
