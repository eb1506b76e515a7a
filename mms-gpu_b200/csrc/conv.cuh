// Exact potential as a convolution: the sum phi_i = sum_j rho_j dV / |r_i - r_j|
// (fmm_calc.cu:412-461) depends on the integer offset alone, so it is a 3-D
// aperiodic convolution with the even kernel G = dV/|r|, G(0) = 0.  It is
// evaluated in FP64 by zero-padded Fourier transforms over x and y (the few
// layers are summed directly): the same sum as the pair loop's to FP64
// rounding, in O(N log N) instead of O(N^2) operations.
//
//   rows    two real rows (y, y + 1) of a layer are one complex transform of
//           length nx >= 2 X - 1; their half spectra (hx = nx/2 + 1 values,
//           each doubled) are separated and stored by column [kx][z][y]
//   columns per kx the Z columns are transformed over y (length ny >= 2 Y - 1),
//           multiplied per ky by the Z x Z matrix Ghat[|z - z'|] (real, because
//           G is even) and transformed back; rows y < Y are kept
//   rows    two half spectra are joined into one complex transform back,
//           phi is rounded to FP32
//
// Transforms are Stockham passes of radix 3, 4, 5, 6, 8, 10, 12 or 16, one butterfly per
// thread and pass, in place in shared memory (every thread reads its inputs
// into registers, the CTA synchronises, then every thread writes), the first
// pass reading its source and the last writing its destination where that can
// be.  The lengths are a fixed list, each with its radices at compile time
// (with run-time radices the passes spilled and the index arithmetic took as
// long as the butterflies).  The inverse is the forward transform with real
// and imaginary parts exchanged before and after.
//
// The columns are kept in device memory, a launch per pass (conv.cu for a
// context's grid, ens.cu for all instances of an ensemble).
//
// A charge that is not finite leaves no value of the potential finite.
#pragma once

#include "mms_internal.cuh"

namespace mmsconv {

constexpr int ZMAX = 8;      // most layers of a column (held in registers)

// A transform of the product of the radices, the largest first: 16 only there,
// where no twiddles are held beside its 16 elements.
template <int R0, int R1, int R2 = 1, int R3 = 1>
struct Radices {
    static constexpr int n = R0 * R1 * R2 * R3;
    static constexpr int last = R3 > 1 ? R3 : R2 > 1 ? R2 : R1;
    static constexpr int rmin = R0 < R1 ? (R0 < last ? R0 : last) : (R1 < last ? R1 : last);
    static constexpr int mmax = n / rmin;  // butterflies of its widest pass
    // padded position of element i: i + (i >> shift) keeps the stores of the
    // first pass (R0 apart) on different banks
    static constexpr int shift = R0 == 16 ? 4 : R0 == 8 ? 3 : 2;
    static constexpr int stride = (n + (n >> shift)) | 1;  // odd: lanes on different transforms, different banks
};

// The lengths, in two sets of radices.  Single grids take small ones: many
// threads with little each, so that a launch of a few CTAs ends soon (64 x 64 x 3:
// 77 us a step against 89 with the other set).  Batches take few passes with
// balanced radices, at most 64 butterflies each (the threads of their CTAs; none for
// 384), and stop at 512 (512 instances: 602 us a step against 710).
constexpr int NPLANS = 19, NBATCH = 12;
template <class F>
void with_plan(int id, F &&f)
{
    switch (id) {
    case 0: f(Radices<4, 4>{}); break;          // 16
    case 1: f(Radices<8, 4>{}); break;          // 32
    case 2: f(Radices<4, 4, 3>{}); break;       // 48
    case 3: f(Radices<8, 8>{}); break;          // 64
    case 4: f(Radices<4, 5, 4>{}); break;       // 80
    case 5: f(Radices<8, 4, 3>{}); break;       // 96
    case 6: f(Radices<8, 4, 4>{}); break;       // 128
    case 7: f(Radices<8, 5, 4>{}); break;       // 160
    case 8: f(Radices<8, 8, 3>{}); break;       // 192
    case 9: f(Radices<8, 8, 4>{}); break;       // 256
    case 10: f(Radices<8, 8, 5>{}); break;      // 320
    case 11: f(Radices<16, 8, 3>{}); break;     // 384
    case 12: f(Radices<8, 8, 8>{}); break;      // 512
    case 13: f(Radices<16, 8, 5>{}); break;     // 640
    case 14: f(Radices<8, 8, 4, 3>{}); break;   // 768
    case 15: f(Radices<16, 8, 8>{}); break;     // 1024
    case 16: f(Radices<8, 8, 8, 3>{}); break;   // 1536
    case 17: f(Radices<8, 8, 8, 4>{}); break;   // 2048
    case 18: f(Radices<8, 8, 8, 8>{}); break;   // 4096
    }
}

#define MMS_CONV_BATCH_PLANS(f)                              \
    case 0: f(Radices<4, 4>{}); break;                       \
    case 1: f(Radices<8, 4>{}); break;                       \
    case 2: f(Radices<8, 6>{}); break;                       \
    case 3: f(Radices<8, 8>{}); break;                       \
    case 4: f(Radices<8, 10>{}); break;                      \
    case 5: f(Radices<8, 12>{}); break;                      \
    case 6: f(Radices<16, 8>{}); break;                      \
    case 7: f(Radices<16, 10>{}); break;                     \
    case 8: f(Radices<8, 8, 3>{}); break;                    \
    case 9: f(Radices<8, 8, 4>{}); break;                    \
    case 10: f(Radices<8, 8, 5>{}); break;                   \
    case 11: f(Radices<8, 8, 8>{}); break;

template <class F>
void with_batch_plan_host(int id, F &&f)
{
    switch (id) {
        MMS_CONV_BATCH_PLANS(f)
    }
}
// in one kernel: a CTA's length is its instance's
template <class F>
__device__ __forceinline__ void with_batch_plan(int id, F &&f)
{
    switch (id) {
        MMS_CONV_BATCH_PLANS(f)
    }
}

struct FftPlan {
    int id, n, stride, mmax;
};

// row pairs per CTA of `threads`, at most `most` (4: a 128-byte run of each column)
template <class PL>
__host__ __device__ constexpr int row_pairs(int threads, int most)
{
    return threads / PL::mmax < 1 ? 1 : threads / PL::mmax > most ? most : threads / PL::mmax;
}

// One grid's convolution with the column store in device memory
struct ConvDev {
    int X, Y, Z, hx, hy;
    int ys, cs;      // elements between layers / columns in the column store
    int fb, cpg;     // row pairs and columns per CTA
    FftPlan px, py;
    const double2 *twx, *twy;  // exp(-2 pi i k / n), k < n
    const double *G;           // [kx < hx][|dz| < Z][ky < hy], scaled by 1 / (2 nx ny)
};

__host__ __device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a
__host__ __device__ __forceinline__ double2 scl(double s, double2 a) { return make_double2(s * a.x, s * a.y); }

__host__ __device__ __forceinline__ void dft4(double2 &a0, double2 &a1, double2 &a2, double2 &a3)
{
    const double2 t0 = a0 + a2, t1 = a0 - a2, t2 = a1 + a3, t3 = mul_mi(a1 - a3);
    a0 = t0 + t2;
    a1 = t1 + t3;
    a2 = t0 - t2;
    a3 = t1 - t3;
}

// v <- DFT of v, natural order in and out
template <int R>
__host__ __device__ __forceinline__ void dft(double2 *v);

template <>
__host__ __device__ __forceinline__ void dft<3>(double2 *v)
{
    constexpr double S = 0.86602540378443864676;  // sin(pi / 3)
    const double2 t = v[1] + v[2], s = mul_mi(scl(S, v[1] - v[2]));
    const double2 m = make_double2(v[0].x - 0.5 * t.x, v[0].y - 0.5 * t.y);
    v[0] = v[0] + t;
    v[1] = m + s;
    v[2] = m - s;
}
template <>
__host__ __device__ __forceinline__ void dft<4>(double2 *v)
{
    dft4(v[0], v[1], v[2], v[3]);
}
template <>
__host__ __device__ __forceinline__ void dft<5>(double2 *v)
{
    constexpr double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr double S1 = 0.95105651629515357212, S2 = 0.58778525229247312917;   // sin(2 pi / 5), sin(4 pi / 5)
    const double2 t1 = v[1] + v[4], t2 = v[2] + v[3], t3 = v[1] - v[4], t4 = v[2] - v[3];
    const double2 m1 = make_double2(v[0].x + C1 * t1.x + C2 * t2.x, v[0].y + C1 * t1.y + C2 * t2.y);
    const double2 m2 = make_double2(v[0].x + C2 * t1.x + C1 * t2.x, v[0].y + C2 * t1.y + C1 * t2.y);
    const double2 s1 = mul_mi(make_double2(S1 * t3.x + S2 * t4.x, S1 * t3.y + S2 * t4.y));
    const double2 s2 = mul_mi(make_double2(S2 * t3.x - S1 * t4.x, S2 * t3.y - S1 * t4.y));
    v[0] = v[0] + t1 + t2;
    v[1] = m1 + s1;
    v[4] = m1 - s1;
    v[2] = m2 + s2;
    v[3] = m2 - s2;
}
// N1 N2, coprime: element N2 i1 + N1 i2 (mod n) to output k with k = k1 (mod
// N1) and k = k2 (mod N2), no twiddles (Good 1958)
template <int N1, int N2>
__host__ __device__ __forceinline__ void dft_coprime(double2 *v)
{
    constexpr int n = N1 * N2;
    double2 t[N2][N1];
#pragma unroll
    for (int i2 = 0; i2 < N2; i2++) {
#pragma unroll
        for (int i1 = 0; i1 < N1; i1++) t[i2][i1] = v[(N2 * i1 + N1 * i2) % n];
        dft<N1>(t[i2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; k1++) {
        double2 u[N2];
#pragma unroll
        for (int i2 = 0; i2 < N2; i2++) u[i2] = t[i2][k1];
        dft<N2>(u);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++)
#pragma unroll
            for (int k = k1; k < n; k += N1)
                if (k % N2 == k2) v[k] = u[k2];  // the output with these residues
    }
}
template <>
__host__ __device__ __forceinline__ void dft<2>(double2 *v)
{
    const double2 a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
}
template <>
__host__ __device__ __forceinline__ void dft<6>(double2 *v) { dft_coprime<2, 3>(v); }
template <>
__host__ __device__ __forceinline__ void dft<10>(double2 *v) { dft_coprime<2, 5>(v); }
template <>
__host__ __device__ __forceinline__ void dft<12>(double2 *v) { dft_coprime<4, 3>(v); }

// R = 4, 8, 16: what follows the sub-transforms of 4 over v[j], v[j + R/4], ...
template <int R>
__host__ __device__ __forceinline__ void dft_rest(double2 *v);
template <>
__host__ __device__ __forceinline__ void dft_rest<4>(double2 *) {}
template <>
__host__ __device__ __forceinline__ void dft_rest<8>(double2 *v)
{
    constexpr double H = 0.70710678118654752440;
    const double2 o0 = v[1], o2 = mul_mi(v[5]);
    const double2 o1 = make_double2(H * (v[3].x + v[3].y), H * (v[3].y - v[3].x));
    const double2 o3 = make_double2(H * (v[7].y - v[7].x), -H * (v[7].x + v[7].y));
    const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = e0 + o0;
    v[4] = e0 - o0;
    v[1] = e1 + o1;
    v[5] = e1 - o1;
    v[2] = e2 + o2;
    v[6] = e2 - o2;
    v[3] = e3 + o3;
    v[7] = e3 - o3;
}
template <>
__host__ __device__ __forceinline__ void dft_rest<16>(double2 *v)
{
    constexpr double H = 0.70710678118654752440, C = 0.92387953251128675613, S = 0.38268343236508977173;
    // v[j + 4 k] is output k of sub-transform j: times exp(-2 pi i j k / 16)
    v[5] = cmul(v[5], make_double2(C, -S));
    v[6] = make_double2(H * (v[6].x + v[6].y), H * (v[6].y - v[6].x));
    v[7] = cmul(v[7], make_double2(S, -C));
    v[9] = make_double2(H * (v[9].x + v[9].y), H * (v[9].y - v[9].x));
    v[10] = mul_mi(v[10]);
    v[11] = make_double2(H * (v[11].y - v[11].x), -H * (v[11].x + v[11].y));
    v[13] = cmul(v[13], make_double2(S, -C));
    v[14] = make_double2(H * (v[14].y - v[14].x), -H * (v[14].x + v[14].y));
    v[15] = cmul(v[15], make_double2(-C, S));
#pragma unroll
    for (int k = 0; k < 4; k++) dft4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    // v[4 k + l] is output k + 4 l: transpose
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int l = k + 1; l < 4; l++) {
            const double2 t = v[4 * k + l];
            v[4 * k + l] = v[4 * l + k];
            v[4 * l + k] = t;
        }
}

template <>
__host__ __device__ __forceinline__ void dft<8>(double2 *v)
{
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    dft_rest<8>(v);
}
template <>
__host__ __device__ __forceinline__ void dft<16>(double2 *v)
{
#pragma unroll
    for (int j = 0; j < 4; j++) dft4(v[j], v[j + 4], v[j + 8], v[j + 12]);
    dft_rest<16>(v);
}

// DFT of v with the upper half of its inputs zero (the padding of a first pass)
template <int R>
__host__ __device__ __forceinline__ void dft_padded(double2 *v)
{
    if constexpr (R == 4 || R == 8 || R == 16) {
        constexpr int H = R / 4;  // sub-transforms of 4, of which two inputs are not zero
#pragma unroll
        for (int j = 0; j < H; j++) {
            const double2 a = v[j], b = v[j + H], c = mul_mi(b);
            v[j] = a + b;
            v[j + H] = a + c;
            v[j + 2 * H] = a - b;
            v[j + 3 * H] = a - c;
        }
        dft_rest<R>(v);
    } else {
#pragma unroll
        for (int q = R / 2; q < R; q++) v[q] = make_double2(0.0, 0.0);
        dft<R>(v);
    }
}

// host side (conv.cu)
// dims, plans and layout of a grid (batch: with the batches' radices) for CTAs
// of `threads` with at most `pairs` row pairs; false where it has none.  *smem:
// what a row or column CTA needs.
bool conv_layout(ConvDev &c, int X, int Y, int Z, bool batch, int threads, int pairs, size_t *smem);
// bytes of the twiddles and Ghat for these lengths and layers, and of the
// scratch their construction needs
size_t conv_table_bytes(const ConvDev &c);
size_t conv_table_scratch(const ConvDev &c);
// builds them in `tab` (256-byte aligned); scratch is free once the stream is
// past the launches
int conv_build_tables(ConvDev &c, void *tab, double *scratch, double dx, double dy, double dz, cudaStream_t st,
                      int64_t *launches);

// One Stockham pass of nf transforms, one butterfly per thread (nf n / R <=
// blockDim): ld(f) gives a reader of transform f's elements, st(f) a writer.
// sync: between the reads and the writes (in-place passes; one with another
// source or destination does without).  LOW_IN: elements from n / 2 up are
// padding and not read; LOW_OUT: those of the result are not wanted.  FB > 0:
// consecutive threads take the same butterfly of FB consecutive transforms
// (whose elements the source holds side by side), else consecutive ones of one.
template <class PL, int NS, int R, bool LOW_IN, bool LOW_OUT, int FB, class LD, class ST>
__device__ __forceinline__ void fft_pass(const double2 *__restrict__ tw, int nf, bool sync, LD ld, ST st)
{
    constexpr int m = PL::n / R;
    const int f = FB > 0 ? threadIdx.x % (FB > 0 ? FB : 1) : threadIdx.x / m;
    const int b = FB > 0 ? threadIdx.x / (FB > 0 ? FB : 1) : threadIdx.x % m;
    const bool on = f < nf && b < m;
    double2 v[R];
    const int k = b % NS, base = (b / NS) * NS * R + k;
    if (on) {
        const auto get = ld(f);
#pragma unroll
        for (int q = 0; q < (LOW_IN ? R / 2 : R); q++) v[q] = get(b + q * m);
        if constexpr (NS > 1) {
            const int step = k * (m / NS);  // n / (NS R)
#pragma unroll
            for (int q = 1; q < R; q++) v[q] = cmul(v[q], __ldg(&tw[q * step]));
        }
        if constexpr (LOW_IN)
            dft_padded<R>(v);
        else
            dft<R>(v);
    }
    if (sync) __syncthreads();
    if (on) {
        const auto put = st(f);
#pragma unroll
        for (int q = 0; q < R; q++)
            if (!LOW_OUT || 2 * q * NS < PL::n) put(base + q * NS, v[q]);
    }
}

// nf transforms of source ld into buf (TO_BUF) or st.  buf holds nf padded
// transforms and is not in use when called, unless ld reads it (IN_PLACE:
// element i of transform f at its own place); the caller synchronises
// afterwards.  A source other than buf has n / 2 elements at most, and so has
// the result that goes to st.  FB: of the first pass.
template <bool TO_BUF, bool IN_PLACE, int FB, int R0, int R1, int R2, int R3, class LD, class ST>
__device__ __forceinline__ void fft_batch(Radices<R0, R1, R2, R3>, const double2 *tw, double2 *buf, int nf, LD ld, ST st)
{
    using PL = Radices<R0, R1, R2, R3>;
    auto bld = [=](int f) {
        const double2 *p = buf + f * PL::stride;
        return [=](int i) { return p[i + (i >> PL::shift)]; };
    };
    auto bst = [=](int f) {
        double2 *p = buf + f * PL::stride;
        return [=](int i, double2 v) { p[i + (i >> PL::shift)] = v; };
    };
    fft_pass<PL, 1, R0, TO_BUF && !IN_PLACE, false, FB>(tw, nf, IN_PLACE, ld, bst);
    __syncthreads();
    if constexpr (R2 > 1) {
        fft_pass<PL, R0, R1, false, false, 0>(tw, nf, true, bld, bst);
        __syncthreads();
    }
    if constexpr (R3 > 1) {
        fft_pass<PL, R0 * R1, R2, false, false, 0>(tw, nf, true, bld, bst);
        __syncthreads();
    }
    if constexpr (TO_BUF)
        fft_pass<PL, PL::n / PL::last, PL::last, false, false, 0>(tw, nf, true, bld, bst);
    else
        fft_pass<PL, PL::n / PL::last, PL::last, false, true, 0>(tw, nf, false, bld, st);
}

// Rows forward for pairs p0 .. p0 + np - 1 (np <= FB; pair p: layer p / hp,
// rows y0 = 2 (p % hp) and y0 + 1): src(z, y) gives a reader of the charges of
// a row, read(x, inside) (x is a cell of the row either way, so that every load
// can be in flight at once), col(kx) the column store of kx.  buf is free on return.
template <int FB, class PL, class SRC, class COL>
__device__ __forceinline__ void rows_forward(PL pl, const ConvDev &c, double2 *buf, int p0, int np, SRC src, COL col)
{
    const int hp = (c.Y + 1) >> 1;
    fft_batch<true, false, 0>(
        pl, c.twx, buf, np,
        [&](int f) {
            const int p = p0 + f, z = p / hp, y = 2 * (p - z * hp), X = c.X;
            const bool two = y + 1 < c.Y;
            const auto ra = src(z, y), rb = src(z, two ? y + 1 : y);
            return [=](int x) {
                const bool in = x < X;
                const int xx = in ? x : X - 1;
                const double a = (double)ra(xx, in), b = (double)rb(xx, in && two);
                return make_double2(in ? a : 0.0, in && two ? b : 0.0);
            };
        },
        [](int) { return [](int, double2) {}; });
    __syncthreads();
    for (int e = threadIdx.x; e < FB * (PL::n / 2 + 1); e += blockDim.x) {
        const int k = e / FB, f = e % FB;
        if (f >= np) continue;
        const int kn = k ? PL::n - k : 0;
        const double2 *t = buf + f * PL::stride;
        const double2 a = t[k + (k >> PL::shift)], b = t[kn + (kn >> PL::shift)];
        const int p = p0 + f, z = p / hp, y = 2 * (p - z * hp);
        double2 *d = col(k) + z * c.ys + y;
        d[0] = make_double2(a.x + b.x, a.y - b.y);
        d[1] = make_double2(a.y + b.y, b.x - a.x);  // (of an odd Y's last pair: the padding row)
    }
    __syncthreads();
}

// The layers' spectra of nc columns times Ghat, real and imaginary parts
// exchanged (the next transform goes back).  ZM: the layers, or their bound.
template <class PL, int ZM, class KX>
__device__ __forceinline__ void times_kernel(const ConvDev &c, double2 *buf, int nc, KX kx)
{
    const int Z = ZM == ZMAX ? c.Z : ZM;
    for (int e = threadIdx.x; e < nc * PL::n; e += blockDim.x) {
        const int j = e / PL::n, ky = e % PL::n, kk = min(ky, PL::n - ky);
        const double *g = c.G + (long long)kx(j) * Z * c.hy + kk;
        double2 *v = buf + j * Z * PL::stride + ky + (ky >> PL::shift);
        double gv[ZM];
        double2 a[ZM];
#pragma unroll
        for (int z = 0; z < ZM; z++)
            if (z < Z) {
                gv[z] = __ldg(g + z * c.hy);
                a[z] = v[z * PL::stride];
            }
#pragma unroll
        for (int z = 0; z < ZM; z++)
            if (z < Z) {
                double2 s = make_double2(0.0, 0.0);
#pragma unroll
                for (int w = 0; w < ZM; w++)
                    if (w < Z) {
                        const double gg = gv[z > w ? z - w : w - z];
                        s.x = fma(gg, a[w].x, s.x);
                        s.y = fma(gg, a[w].y, s.y);
                    }
                v[z * PL::stride] = make_double2(s.y, s.x);
            }
    }
}

// The Z columns of each of nc columns (col(j), kx(j)): forward, times Ghat,
// back, in the column store.  nc Z padded transforms in buf; groups of whole
// transforms that fit the CTA one butterfly per thread.
template <class PL, class COL, class KX>
__device__ __forceinline__ void columns(PL pl, const ConvDev &c, double2 *buf, int nc, COL col, KX kx)
{
    const int Z = c.Z, Y = c.Y, ys = c.ys;
    const int nf = nc * Z, per = min(nf, max(1, (int)blockDim.x / PL::mmax));
    for (int f0 = 0; f0 < nf; f0 += per)
        fft_batch<true, false, 0>(
            pl, c.twy, buf + f0 * PL::stride, min(per, nf - f0),
            [&](int f) {
                const int j = (f0 + f) / Z, z = f0 + f - j * Z;
                const double2 *p = col(j) + z * ys;
                return [=](int y) {
                    const double2 a = p[min(y, Y - 1)];
                    return make_double2(y < Y ? a.x : 0.0, y < Y ? a.y : 0.0);
                };
            },
            [](int) { return [](int, double2) {}; });
    __syncthreads();
    switch (Z) {
    case 1: times_kernel<PL, 1>(c, buf, nc, kx); break;
    case 2: times_kernel<PL, 2>(c, buf, nc, kx); break;
    case 3: times_kernel<PL, 3>(c, buf, nc, kx); break;
    case 4: times_kernel<PL, 4>(c, buf, nc, kx); break;
    default: times_kernel<PL, ZMAX>(c, buf, nc, kx); break;
    }
    __syncthreads();
    for (int f0 = 0; f0 < nf; f0 += per) {
        double2 *b0 = buf + f0 * PL::stride;
        fft_batch<false, true, 0>(
            pl, c.twy, b0, min(per, nf - f0),
            [=](int f) {
                const double2 *p = b0 + f * PL::stride;
                return [=](int y) { return p[y + (y >> PL::shift)]; };
            },
            [&](int f) {
                const int j = (f0 + f) / Z, z = f0 + f - j * Z;
                double2 *p = col(j) + z * ys;
                return [=](int y, double2 v) {
                    if (y < Y) p[y] = make_double2(v.y, v.x);
                };
            });
    }
    __syncthreads();
}

// Rows back for pairs p0 .. p0 + np - 1: dst(z, y) gives a writer of phi's row.
template <int FB, class PL, class COL, class DST>
__device__ __forceinline__ void rows_back(PL pl, const ConvDev &c, double2 *buf, int p0, int np, COL col, DST dst)
{
    const int hp = (c.Y + 1) >> 1;
    fft_batch<false, false, FB>(
        pl, c.twx, buf, np,
        [&](int f) {
            const int p = p0 + f, z = p / hp, y = 2 * (p - z * hp), o = z * c.ys + y;
            return [=](int i) {
                const bool up = 2 * i > PL::n;
                const double2 *d = col(up ? PL::n - i : i) + o;
                const double2 a = d[0], b = d[1];
                // a + i b (conjugates above n / 2), parts exchanged
                return up ? make_double2(b.x - a.y, a.x + b.y) : make_double2(a.y + b.x, a.x - b.y);
            };
        },
        [&](int f) {
            const int p = p0 + f, z = p / hp, y = 2 * (p - z * hp), X = c.X;
            const bool two = y + 1 < c.Y;
            const auto ra = dst(z, y), rb = dst(z, two ? y + 1 : y);
            return [=](int x, double2 v) {
                if (x >= X) return;
                ra(x, (float)v.y);
                if (two) rb(x, (float)v.x);
            };
        });
    __syncthreads();
}

}  // namespace mmsconv
