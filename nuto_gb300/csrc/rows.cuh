// CSR rows from element matrices, the second half of every element-matrix tangent (FP32: fused.cu, FP64: tangent64.cu).
//
// An element matrix is ND slabs, one per local node a: NR rows (a's displacement components, then its eeq row) x NC columns
// (the displacement components of b = 0..ND-1, b-major, then the eeq of b = 0..ND-1). A group of lanes owns one displacement
// node: lane = slab column; the slabs of the node's cells are added in ascending cell order into a shared copy of the node's
// rows at the ranks of b (a cell's b are distinct nodes: no conflicts) and the rows are stored once. No atomics: the values
// are bitwise reproducible.
//
// Bound by the latency of the chain node -> cells -> slab. It is kept to three dependent loads: the node's plan (rows,
// block offsets, cell list: one 64-byte record), the slab numbers and packed ranks of a batch of 4 cells, their slabs.
// The rows are kept interleaved (the eeq row has the positions of the displacement rows): one vector access per column instead
// of one per row. FP32 Hex8 gradient damage at 48^3: 160 us with row
// pointers, cell indices and block offsets read one after the other, 139 us with the plan, 118 us interleaved (DRAM floor
// 95 us; 81 % of the shared-memory wavefronts). Quad4 gradient damage (16 lanes per node) 70 -> 30 us for 71 k nodes.
#pragma once

#include "internal.cuh"

namespace nuto_gpu
{

constexpr int kRowsCap = 128; // values per row: 32 neighbour nodes of [u | eeq] in 3D

template <int DIM, int ND, bool GD>
struct Slab
{
    static constexpr int nr = DIM + (GD ? 1 : 0);      // rows per local node
    static constexpr int nc = ND * DIM + (GD ? ND : 0); // columns per row
    static constexpr int size = nr * nc;
    // lanes per node: the columns rounded up to a power of two
    static constexpr int lanes = nc > 16 ? 32 : (nc > 8 ? 16 : 8);
};

// One value of every row of a node at one position, read and written as one vector
template <typename T, int NR>
struct alignas(NR == 2 ? 2 * sizeof(T) : 16) RowVec
{
    static constexpr int n = NR == 3 ? 4 : NR;
    T v[n];
};

// The rows of a node have the same positions and are kept interleaved: one vector access per column updates all of them
template <typename T, int DIM, int ND, bool GD, int W>
__global__ void __launch_bounds__(W * 32) k_rows_from_slabs(RowPlanArgs P, const T* __restrict__ em, T* __restrict__ vals)
{
    using S = Slab<DIM, ND, GD>;
    constexpr int NR = S::nr, NC = S::nc, LPN = S::lanes, NPW = 32 / LPN, CB = 4;
    using V = RowVec<T, NR>;
    __shared__ V sRowAll[W * NPW][kRowsCap];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane / LPN, col = lane % LPN;
    PdlWait();
    const int64_t a = P.nodeFirst + (static_cast<int64_t>(blockIdx.x) * W + wid) * NPW + grp;
    V* sVec = sRowAll[wid * NPW + grp];
    RowPlan p{};
    if (a < P.nodeLast)
        p = P.plan[a]; // p.cells = 0 beyond the last node: nothing to add or store
    for (int i = col; i < p.len; i += LPN)
        sVec[i] = V{};
    const bool ucol = col < ND * DIM;
    const int myB = col < NC ? (ucol ? col / DIM : col - ND * DIM) : 0;
    const int myL = ucol ? col % DIM : 0;
    int most = p.cells;
    if (NPW > 1)
    {
#pragma unroll
        for (int o = LPN; o < 32; o <<= 1)
            most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    }
    __syncwarp();
    for (int kb = 0; kb < most; kb += CB)
    {
        uint32_t slab[CB], word[CB];
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            const bool on = kb + c < p.cells;
            slab[c] = on ? P.slab[NG_IDX(p.first + kb + c, P.nEntries, 77)] : 0u;
            word[c] = on ? P.packed[NG_IDX((p.first + kb + c) * ND + myB, P.nEntries * ND, 77)] : 0u;
        }
        T v[CB][NR];
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            const bool on = kb + c < p.cells && col < NC;
            const T* src = em + NG_IDX(slab[c], P.nEntries, 78) * static_cast<int64_t>(S::size) + col;
#pragma unroll
            for (int r = 0; r < NR; ++r)
                v[c][r] = on ? src[r * NC] : T(0);
        }
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            if (kb + c < p.cells && col < NC)
            {
                const int rank = ucol ? word[c] & 0xff : word[c] >> 8;
                V& row = sVec[NG_IDX(ucol ? p.bU + DIM * rank + myL : p.bE + rank, kRowsCap, 79)];
                V x = row;
#pragma unroll
                for (int k = 0; k < NR; ++k)
                    x.v[k] += v[c][k];
                row = x;
            }
            __syncwarp();
        }
    }
    for (int i = col; i < p.len; i += LPN)
    {
        const V x = sVec[i];
#pragma unroll
        for (int k = 0; k < DIM; ++k)
            vals[NG_IDX(p.rowU + static_cast<int64_t>(k) * p.len + i, P.nnz, 75)] = x.v[k];
        if (GD)
            vals[NG_IDX(p.rowE + i, P.nnz, 75)] = x.v[DIM];
    }
}

// The gather for displacement cells whose slabs are wider than a warp (Hex20: 3 rows x 60 columns): one warp per node, lane l
// the columns l and l + 32. The rows of a node (up to kRowsCapWide values) are interleaved in shared memory. FP32 24^3: 112 us
// with byte ranks, cell indices and row pointers read one after the other, 80 us with the plan.
constexpr int kRowsCapWide = 256;

template <typename T, int ND, int W>
__global__ void __launch_bounds__(W * 32) k_rows_from_wide_slabs(RowPlanArgs P, const T* __restrict__ em,
                                                                T* __restrict__ vals)
{
    constexpr int NC = 3 * ND, CB = 2;
    static_assert(NC > 32 && NC <= 64, "two columns per lane");
    using V = RowVec<T, 3>;
    extern __shared__ __align__(16) unsigned char smW[];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    V* row = reinterpret_cast<V*>(smW) + wid * kRowsCapWide;
    PdlWait();
    const int64_t a = static_cast<int64_t>(blockIdx.x) * W + wid;
    if (a >= P.nodeLast)
        return; // the whole warp leaves; only warp-level synchronisation follows
    const RowPlan p = P.plan[a];
    for (int i = lane; i < p.len; i += 32)
        row[i] = V{};
    const bool second = lane + 32 < NC;
    const int b0 = lane / 3, l0 = lane % 3, b1 = second ? (lane + 32) / 3 : 0, l1 = (lane + 32) % 3;
    __syncwarp();
    for (int kb = 0; kb < p.cells; kb += CB)
    {
        uint32_t slab[CB], w0[CB], w1[CB];
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            const int64_t kc = p.first + (kb + c < p.cells ? kb + c : kb);
            slab[c] = P.slab[NG_IDX(kc, P.nEntries, 77)];
            w0[c] = P.packed[NG_IDX(kc * ND + b0, P.nEntries * ND, 77)];
            w1[c] = P.packed[NG_IDX(kc * ND + b1, P.nEntries * ND, 77)];
        }
        T v[CB][2][3];
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            const T* src = em + NG_IDX(slab[c], P.nEntries, 78) * static_cast<int64_t>(3 * NC) + lane;
#pragma unroll
            for (int r = 0; r < 3; ++r)
            {
                v[c][0][r] = src[r * NC];
                v[c][1][r] = second ? src[r * NC + 32] : T(0);
            }
        }
#pragma unroll
        for (int c = 0; c < CB; ++c)
        {
            if (kb + c < p.cells)
            {
                V& x0 = row[NG_IDX(p.bU + 3 * static_cast<int>(w0[c] & 0xff) + l0, kRowsCapWide, 79)];
                V t = x0;
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    t.v[r] += v[c][0][r];
                x0 = t;
                if (second)
                {
                    V& x1 = row[NG_IDX(p.bU + 3 * static_cast<int>(w1[c] & 0xff) + l1, kRowsCapWide, 79)];
                    V s = x1;
#pragma unroll
                    for (int r = 0; r < 3; ++r)
                        s.v[r] += v[c][1][r];
                    x1 = s;
                }
            }
            __syncwarp();
        }
    }
    for (int i = lane; i < p.len; i += 32)
    {
        const V x = row[i];
#pragma unroll
        for (int k = 0; k < 3; ++k)
            vals[NG_IDX(p.rowU + static_cast<int64_t>(k) * p.len + i, P.nnz, 75)] = x.v[k];
    }
}

template <typename T, int ND>
inline void LaunchWideRows(Ctx& c, const RowPlanArgs& all, int64_t nNodes, const T* em, T* vals)
{
    constexpr int W = 4;
    RowPlanArgs P = all;
    P.nodeFirst = 0;
    P.nodeLast = nNodes;
    constexpr size_t smem = static_cast<size_t>(W) * kRowsCapWide * sizeof(RowVec<T, 3>);
    static_assert(smem <= 48 * 1024, "no opt-in needed");
    NG_CUDA(LaunchPdl(k_rows_from_wide_slabs<T, ND, W>, dim3(static_cast<unsigned>((nNodes + W - 1) / W)), dim3(W * 32), smem,
                      c.stream, P, em, vals));
    AfterLaunch(c, "k_rows_from_wide_slabs");
    c.stats.kernel_launches += 1;
}

// Launches the gather for the displacement nodes first .. last - 1.
template <typename T, int DIM, int ND, bool GD, int W>
inline void LaunchRows(Ctx& c, const RowPlanArgs& all, int64_t first, int64_t last, const T* em, T* vals)
{
    RowPlanArgs P = all;
    P.nodeFirst = first;
    P.nodeLast = last;
    constexpr int perBlock = W * (32 / Slab<DIM, ND, GD>::lanes);
    if (last <= first)
        return;
    const dim3 grid(static_cast<unsigned>((last - first + perBlock - 1) / perBlock));
    NG_CUDA(LaunchEx(true, c.carveout, k_rows_from_slabs<T, DIM, ND, GD, W>, grid, dim3(W * 32), 0, c.stream, P, em, vals));
    AfterLaunch(c, "k_rows_from_slabs");
    c.stats.kernel_launches += 1;
}

} // namespace nuto_gpu
