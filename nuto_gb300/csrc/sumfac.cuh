// Tensor-product (sum-factorised) evaluation of linear fields at the two-point Gauss rule: Quad4 cells with 2 x 2 and
// Hex8 cells with 2 x 2 x 2 points, and the transposes of these maps (InterpolationQuadLinear.cpp:37-80,
// InterpolationBrickLinear.cpp:37-132 in the local node order, points with the first coordinate running fastest).
//
// In one direction the shape values at the points -1/sqrt(3), 1/sqrt(3) are [[p, m], [m, p]] with p = (1 + 1/sqrt(3)) / 2
// and m = (1 - 1/sqrt(3)) / 2, and the derivatives are -1/2, 1/2 at both points. Divided by m the interpolation is
// [[r, 1], [1, r]] with r = p / m = 2 + sqrt(3): one multiply-add per value. A field's gradient at the 8 points of a Hex8
// cell then takes 36 operations instead of 192 (its x-derivative does not depend on the x-coordinate of the point, so
// there are 4 values per direction), its values 8 more. The factors m per interpolation are left out here: gradients
// carry 2 / m^(DIM-1) (folded into the cached inverse Jacobian), values 1 / m^DIM.
// The point of it: the FP64 pipe of this part issues 2 lanes per clock and SM, so every FP64 instruction counts.
#pragma once

#include "internal.cuh"

namespace nuto_gpu
{

constexpr double kSfRatio = 3.7320508075688772935;  // r = (1 + g) / (1 - g), g = 1 / sqrt(3)
constexpr double kSfMinor = 0.21132486540518711775; // m = (1 - g) / 2

template <int DIM>
struct SumFac
{
    static constexpr int nd = DIM == 3 ? 8 : 4;          // nodes = points
    static constexpr int ng1 = DIM == 3 ? 4 : 2;         // distinct values of one derivative
    static constexpr int ng = ng1 * DIM;                 // all derivatives of one field
    // gradients: natural derivative = gradScale * the value computed here; values: value = valScale * the computed one
    static constexpr double gradScale = DIM == 3 ? 0.5 * kSfMinor * kSfMinor : 0.5 * kSfMinor;
    static constexpr double valScale = DIM == 3 ? kSfMinor * kSfMinor * kSfMinor : kSfMinor * kSfMinor;
};

// index of derivative j at point q among the ng values (x derivatives first)
template <int DIM>
__host__ __device__ constexpr int SfGradIndex(int j, int q)
{
    if (DIM == 3)
        return j == 0 ? (q >> 1) : (j == 1 ? 4 + ((q >> 2) << 1) + (q & 1) : 8 + (q & 3));
    return j == 0 ? (q >> 1) : 2 + (q & 1);
}

// local node at lattice position i (bit d: position along direction d)
__host__ __device__ constexpr int SfNode(int i)
{
    return (i & 4) + ((i & 2) ? ((i & 1) ? 2 : 3) : (i & 1));
}

// [r, 1; 1, r] applied to a pair
template <typename T>
__device__ __forceinline__ void SfPair(T a, T b, T& oa, T& ob)
{
    const T r = T(kSfRatio);
    oa = r * a + b;
    ob = r * b + a;
}

// nodal values (local node order) -> the ng derivatives and (VAL) the values at the points
template <typename T, int DIM, bool VAL>
__device__ __forceinline__ void SfForward(const T* v, T* g, T* val)
{
    if constexpr (DIM == 2)
    {
        T ix[2][2]; // [y][qx]
#pragma unroll
        for (int y = 0; y < 2; ++y)
            SfPair(v[SfNode(2 * y)], v[SfNode(2 * y + 1)], ix[y][0], ix[y][1]);
        SfPair(v[SfNode(1)] - v[SfNode(0)], v[SfNode(3)] - v[SfNode(2)], g[0], g[1]);
        g[2] = ix[1][0] - ix[0][0];
        g[3] = ix[1][1] - ix[0][1];
        if (VAL)
        {
            SfPair(ix[0][0], ix[1][0], val[0], val[2]);
            SfPair(ix[0][1], ix[1][1], val[1], val[3]);
        }
    }
    else
    {
        T d[2][2];      // x difference [z][y]
        T ix[2][2][2];  // x interpolated [z][y][qx]
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
            for (int y = 0; y < 2; ++y)
            {
                const T a = v[SfNode(4 * z + 2 * y)], b = v[SfNode(4 * z + 2 * y + 1)];
                d[z][y] = b - a;
                SfPair(a, b, ix[z][y][0], ix[z][y][1]);
            }
        T t[2][2]; // [z][qy]
#pragma unroll
        for (int z = 0; z < 2; ++z)
            SfPair(d[z][0], d[z][1], t[z][0], t[z][1]);
#pragma unroll
        for (int qy = 0; qy < 2; ++qy)
            SfPair(t[0][qy], t[1][qy], g[qy], g[2 + qy]);
#pragma unroll
        for (int qx = 0; qx < 2; ++qx)
            SfPair(ix[0][1][qx] - ix[0][0][qx], ix[1][1][qx] - ix[1][0][qx], g[4 + qx], g[6 + qx]);
        T jy[2][2][2]; // x and y interpolated [z][qy][qx]
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
            for (int qx = 0; qx < 2; ++qx)
                SfPair(ix[z][0][qx], ix[z][1][qx], jy[z][0][qx], jy[z][1][qx]);
#pragma unroll
        for (int qy = 0; qy < 2; ++qy)
#pragma unroll
            for (int qx = 0; qx < 2; ++qx)
            {
                g[8 + 2 * qy + qx] = jy[1][qy][qx] - jy[0][qy][qx];
                if (VAL)
                    SfPair(jy[0][qy][qx], jy[1][qy][qx], val[2 * qy + qx], val[4 + 2 * qy + qx]);
            }
    }
}

// The transpose: out[node] = sum over the points of derivative j of node's shape function times F(j, q), plus (VAL) its
// value times V(q) (same factors left out as in SfForward). F and V are read through the accessors.
template <typename T, int DIM, bool VAL, typename FF, typename FV>
__device__ __forceinline__ void SfTranspose(FF&& F, FV&& V, T* out)
{
    if constexpr (DIM == 2)
    {
        T a[2]; // x derivative parts [y]
        SfPair(F(0, 0) + F(0, 1), F(0, 2) + F(0, 3), a[0], a[1]);
        T jy[2][2]; // [y][qx]
#pragma unroll
        for (int qx = 0; qx < 2; ++qx)
        {
            const T s = F(1, qx) + F(1, 2 + qx);
            if (VAL)
            {
                SfPair(V(qx), V(2 + qx), jy[0][qx], jy[1][qx]);
                jy[0][qx] -= s;
                jy[1][qx] += s;
            }
            else
            {
                jy[0][qx] = -s;
                jy[1][qx] = s;
            }
        }
#pragma unroll
        for (int y = 0; y < 2; ++y)
        {
            T o0, o1;
            SfPair(jy[y][0], jy[y][1], o0, o1);
            out[SfNode(2 * y)] = o0 - a[y];
            out[SfNode(2 * y + 1)] = o1 + a[y];
        }
    }
    else
    {
        // x derivatives: summed over qx, interpolated back over z and y -> a[z][y]
        T t[2][2], a[2][2];
#pragma unroll
        for (int qy = 0; qy < 2; ++qy)
            SfPair(F(0, 2 * qy) + F(0, 2 * qy + 1), F(0, 4 + 2 * qy) + F(0, 4 + 2 * qy + 1), t[0][qy], t[1][qy]);
#pragma unroll
        for (int z = 0; z < 2; ++z)
            SfPair(t[z][0], t[z][1], a[z][0], a[z][1]);
        // y derivatives: summed over qy, interpolated back over z -> b[z][qx]
        T b[2][2];
#pragma unroll
        for (int qx = 0; qx < 2; ++qx)
            SfPair(F(1, qx) + F(1, 2 + qx), F(1, 4 + qx) + F(1, 6 + qx), b[0][qx], b[1][qx]);
        // z derivatives and values at [z][qy][qx], then back over y
        T iy[2][2][2]; // [z][y][qx]
#pragma unroll
        for (int qx = 0; qx < 2; ++qx)
        {
            const T s0 = F(2, qx) + F(2, 4 + qx), s1 = F(2, 2 + qx) + F(2, 6 + qx);
            if (VAL)
            {
                T c0[2], c1[2]; // [z]
                SfPair(V(qx), V(4 + qx), c0[0], c0[1]);
                SfPair(V(2 + qx), V(6 + qx), c1[0], c1[1]);
                SfPair(c0[0] - s0, c1[0] - s1, iy[0][0][qx], iy[0][1][qx]);
                SfPair(c0[1] + s0, c1[1] + s1, iy[1][0][qx], iy[1][1][qx]);
            }
            else
            {
                T k0, k1;
                SfPair(s0, s1, k0, k1);
                iy[0][0][qx] = -k0;
                iy[0][1][qx] = -k1;
                iy[1][0][qx] = k0;
                iy[1][1][qx] = k1;
            }
#pragma unroll
            for (int z = 0; z < 2; ++z)
            {
                iy[z][0][qx] -= b[z][qx];
                iy[z][1][qx] += b[z][qx];
            }
        }
#pragma unroll
        for (int z = 0; z < 2; ++z)
#pragma unroll
            for (int y = 0; y < 2; ++y)
            {
                T o0, o1;
                SfPair(iy[z][y][0], iy[z][y][1], o0, o1);
                out[SfNode(4 * z + 2 * y)] = o0 - a[z][y];
                out[SfNode(4 * z + 2 * y + 1)] = o1 + a[z][y];
            }
    }
}

// out[b] = sum over the points q of N_b(q) f[q] up to the factor valScale (the transpose of the interpolation; the
// matrix is symmetric in the lattice order, so the points' order is the lattice order)
template <typename T, int DIM>
__device__ __forceinline__ void SfValuesToNodes(const T* f, T* out)
{
    constexpr int n = SumFac<DIM>::nd;
    T v[n], w[n];
#pragma unroll
    for (int i = 0; i < n; i += 2)
        SfPair(f[i], f[i + 1], v[i], v[i + 1]);
#pragma unroll
    for (int i = 0; i < n; ++i)
        if (!(i & 2))
            SfPair(v[i], v[i + 2], w[i], w[i + 2]);
    if constexpr (DIM == 3)
    {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            SfPair(w[i], w[i + 4], out[SfNode(i)], out[SfNode(i + 4)]);
    }
    else
    {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            out[SfNode(i)] = w[i];
    }
}

// engineering strain from the natural gradients G[c][j] = du_c/dxi_j and the inverse Jacobian J[j][d] = dxi_j/dx_d
template <typename T, int DIM>
__device__ __forceinline__ void StrainFromNatural(const T (&G)[DIM][DIM], const T (&J)[DIM][DIM], T* e)
{
    auto dot = [&](int c, int d, T s) {
#pragma unroll
        for (int j = 0; j < DIM; ++j)
            s += G[c][j] * J[j][d];
        return s;
    };
#pragma unroll
    for (int c = 0; c < DIM; ++c)
        e[c] = dot(c, c, T(0));
    if (DIM == 2)
        e[2] = dot(0, 1, dot(1, 0, T(0)));
    else
    {
        e[3] = dot(1, 2, dot(2, 1, T(0)));
        e[4] = dot(0, 2, dot(2, 0, T(0)));
        e[5] = dot(0, 1, dot(1, 0, T(0)));
    }
}

} // namespace nuto_gpu
