// Per-cell device math shared by the single-grid and the ensemble kernels:
// cell coordinates, the external field table, the effective field from the
// FP32 potential and the FP64 state, and the LLG right-hand side.
#pragma once

#include "mms_internal.cuh"

namespace mmsdev {

// (a grid has at most 2^29 cells: 32-bit divides, a third of the 64-bit ones'
// instructions; 64 x 64 x 3 FMM steps 1.7 % faster, a million-cell field 1.6 %)
__device__ __forceinline__ void cell_xyz(long long i, const GridK &g, int &x, int &y, int &z)
{
    const unsigned c = (unsigned)i, r = c / (unsigned)g.X;
    x = (int)(c - r * g.X);
    z = (int)(r / (unsigned)g.Y);
    y = (int)(r - z * g.Y);
}

// clamped piecewise-linear B(t) table, or the reference's ramp (ode_functions.cpp:61)
__device__ __forceinline__ void hext_at(const PhysK &p, const double *__restrict__ tab, double t, double H[3])
{
    H[0] = H[1] = H[2] = 0.0;
    if (!p.external) return;
    if (p.n_hext == 0) {
        H[0] = p.inv_mu0 * ((t < 1e-9) ? (-0.3 / 1e-9 * t + 0.3) : 0.0);
        return;
    }
    const int n = p.n_hext;
    double b0, b1, b2;
    if (t <= tab[0]) {
        b0 = tab[1]; b1 = tab[2]; b2 = tab[3];
    } else if (t >= tab[4 * (n - 1)]) {
        b0 = tab[4 * (n - 1) + 1]; b1 = tab[4 * (n - 1) + 2]; b2 = tab[4 * (n - 1) + 3];
    } else {
        int k = 0;
        while (k + 1 < n && tab[4 * (k + 1)] < t) k++;
        const double w = (t - tab[4 * k]) / (tab[4 * (k + 1)] - tab[4 * k]);
        b0 = (1 - w) * tab[4 * k + 1] + w * tab[4 * (k + 1) + 1];
        b1 = (1 - w) * tab[4 * k + 2] + w * tab[4 * (k + 1) + 2];
        b2 = (1 - w) * tab[4 * k + 3] + w * tab[4 * (k + 1) + 3];
    }
    H[0] = b0 * p.inv_mu0;
    H[1] = b1 * p.inv_mu0;
    H[2] = b2 * p.inv_mu0;
}

// H_ext at the time ts of an RK4 stage into the slot that the stage reads
__device__ __forceinline__ void put_hext(const PhysK &p, const double *__restrict__ tab, double *__restrict__ tstate,
                                         int stage, double ts)
{
    double he[3];
    hext_at(p, tab, ts, he);
    for (int c = 0; c < 3; c++) tstate[TIME_HEXT + 3 * stage + c] = he[c];
}

// half reciprocal cell sizes 1 / (2 dx), 1 / (2 dy), 1 / (2 dz): the central
// difference weights of div_soa_cell, formed once on the host
struct DivScale {
    double hx, hy, hz;
};
inline DivScale div_scale(double dx, double dy, double dz) { return DivScale{0.5 / dx, 0.5 / dy, 0.5 / dz}; }

// a[i + step] inside the grid, 0 beyond it.  FLAT: the load is unconditional
// (of a[i] beyond the edge), so that a stencil's loads can all be in flight at
// once; the guarded form waits at its branches but measured 1 % faster a step
// where many short kernels fill the chip (256 x 256 x 3 FMM steps, 2,730
// against 2,758 us per 20), the flat one in the ensemble's row pass.
template <bool FLAT, class T>
__device__ __forceinline__ double edge(const T *__restrict__ a, long long i, long long step, bool inside)
{
    if (!FLAT) return inside ? (double)a[i + step] : 0.0;
    const T v = a[i + (inside ? step : 0)];
    return inside ? (double)v : 0.0;
}

// rho = div M at cell i = (x, y, z) of the FP64 SoA state (planes N apart):
// central differences, zero outside the grid (vector_functions.cpp:8-28, in
// FP64), as products with the half reciprocal sizes (no divide on the device)
// rounded one by one (no contraction).  Every kernel that forms rho from the
// state uses this expression, so they agree bit for bit.
template <bool FLAT = false>
__device__ __forceinline__ float div_soa_cell(const double *__restrict__ M, long long i, int x, int y, int z,
                                              const GridK &g, const DivScale &h)
{
    const double *Mx = M, *My = M + g.N, *Mz = M + 2 * g.N;
    const long long sy = g.X, sz = (long long)g.X * g.Y;
    const double x2 = edge<FLAT>(Mx, i, 1, x != g.X - 1), x0 = edge<FLAT>(Mx, i, -1, x != 0);
    const double y2 = edge<FLAT>(My, i, sy, y != g.Y - 1), y0 = edge<FLAT>(My, i, -sy, y != 0);
    const double z2 = edge<FLAT>(Mz, i, sz, z != g.Z - 1), z0 = edge<FLAT>(Mz, i, -sz, z != 0);
    const double a = __dmul_rn(__dsub_rn(x2, x0), h.hx);
    const double b = __dmul_rn(__dsub_rn(y2, y0), h.hy);
    const double c = __dmul_rn(__dsub_rn(z2, z0), h.hz);
    return (float)__dadd_rn(__dadd_rn(a, b), c);
}

// the reference's FP32 divergence (vector_functions.cpp:8-28) at cell i of M (N
// x 3), in its operation order, each operation rounded on its own: its bits
struct DivAos {
    float dx, dy, dz;
};
__device__ __forceinline__ float div_aos_cell(const float *__restrict__ M, long long i, int x, int y, int z,
                                              const GridK &g, const DivAos &d)
{
    const long long sy = g.X, sz = (long long)g.X * g.Y;
    float x2 = (x != g.X - 1) ? M[3 * (i + 1) + 0] : 0.f;
    float x0 = (x != 0) ? M[3 * (i - 1) + 0] : 0.f;
    float y2 = (y != g.Y - 1) ? M[3 * (i + sy) + 1] : 0.f;
    float y0 = (y != 0) ? M[3 * (i - sy) + 1] : 0.f;
    float z2 = (z != g.Z - 1) ? M[3 * (i + sz) + 2] : 0.f;
    float z0 = (z != 0) ? M[3 * (i - sz) + 2] : 0.f;
    float s = __fadd_rn(__fadd_rn(__fdiv_rn(__fsub_rn(x2, x0), d.dx), __fdiv_rn(__fsub_rn(y2, y0), d.dy)),
                        __fdiv_rn(__fsub_rn(z2, z0), d.dz));
    return s * 0.5f;  // (s / 2.0) in double then to float: exact halving
}

// index of cell (x, y, z) in the box-major BF16 charge layout of the
// tensor-core near field, [Z][nby][nbx][8][8] (leaf side 8)
__device__ __forceinline__ long long ntc_index(int x, int y, int z, int nbx, int nby)
{
    return (((long long)z * nby + (y >> 3)) * nbx + (x >> 3)) * 64 + (y & 7) * 8 + (x & 7);
}

// effective field at cell i from phi (FP32) and the FP64 stage state
template <bool FLAT = false>
__device__ __forceinline__ void field_soa(const float *__restrict__ phi, const double *__restrict__ M, long long i,
                                          int x, int y, int z, const GridK &g, const PhysK &p, const double he[3],
                                          double H[3])
{
    const long long sy = g.X, sz = (long long)g.X * g.Y;
    H[0] = he[0];
    H[1] = he[1];
    H[2] = he[2];
    if (p.demag) {
        const double x2 = edge<FLAT>(phi, i, 1, x != g.X - 1), x0 = edge<FLAT>(phi, i, -1, x != 0);
        const double y2 = edge<FLAT>(phi, i, sy, y != g.Y - 1), y0 = edge<FLAT>(phi, i, -sy, y != 0);
        const double z2 = edge<FLAT>(phi, i, sz, z != g.Z - 1), z0 = edge<FLAT>(phi, i, -sz, z != 0);
        H[0] += p.hgx * (x2 - x0);
        H[1] += p.hgy * (y2 - y0);
        H[2] += p.hgz * (z2 - z0);
    }
    if (p.exchange) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double *Mc = M + c * g.N;
            const double m0 = Mc[i];
            const double xp = edge<FLAT>(Mc, i, 1, x != g.X - 1), xm = edge<FLAT>(Mc, i, -1, x != 0);
            const double yp = edge<FLAT>(Mc, i, sy, y != g.Y - 1), ym = edge<FLAT>(Mc, i, -sy, y != 0);
            const double zp = edge<FLAT>(Mc, i, sz, z != g.Z - 1), zm = edge<FLAT>(Mc, i, -sz, z != 0);
            H[c] += (xp + xm - 2 * m0) * p.ecx + (yp + ym - 2 * m0) * p.ecy + (zp + zm - 2 * m0) * p.ecz;
        }
    }
}

// ode_functions.cpp:11-18
__device__ __forceinline__ void llg(const double m[3], const double h[3], const PhysK &p, double k[3])
{
    const double cx = m[1] * h[2] - m[2] * h[1];
    const double cy = m[2] * h[0] - m[0] * h[2];
    const double cz = m[0] * h[1] - m[1] * h[0];
    const double ex = m[1] * cz - m[2] * cy;
    const double ey = m[2] * cx - m[0] * cz;
    const double ez = m[0] * cy - m[1] * cx;
    const double a = p.llg_a;
    k[0] = -p.gamma * cx - a * ex;
    k[1] = -p.gamma * cy - a * ey;
    k[2] = -p.gamma * cz - a * ez;
}

}  // namespace mmsdev
