// Host side of the convolution (conv.cuh): plans, tables, and the launches of
// the exact potential that keep the column store in device memory.
#include <math.h>

#include <algorithm>

#include "conv.cuh"

using namespace mmsconv;

namespace {

constexpr int ROW_PAIRS = 4;              // row pairs per CTA at most: small grids need the CTAs
constexpr int MAX_THREADS = 512;          // threads of a row or column CTA

// tw[k] = exp(-2 pi i k / n)
__global__ void k_conv_twiddle(double2 *__restrict__ tw, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double s, c;
    sincospi(2.0 * k / n, &s, &c);
    tw[k] = make_double2(c, -s);
}

// The even kernel's cosine transform along x, then along y: CTA = one (dz, y)
// row into T[dz][kx][y], then one (kx, dz) column into G.  Offsets beyond
// n / 2 are the mirror images of those below (weight 2; 0 and n / 2 are their
// own); the largest offset of a grid is X - 1 < nx / 2 + 1.
__global__ void k_conv_table_x(double *__restrict__ T, const double2 *__restrict__ tw, int n, int h, int hy, double dx,
                               double dy, double dz)
{
    extern __shared__ double sg[];
    const int y = blockIdx.x % hy, z = blockIdx.x / hy;
    for (int x = threadIdx.x; x < h; x += blockDim.x) {
        const double r2 = x * dx * (x * dx) + y * dy * (y * dy) + z * dz * (z * dz);
        sg[x] = r2 == 0.0 ? 0.0 : dx * dy * dz / sqrt(r2) * (x == 0 || 2 * x == n ? 1.0 : 2.0);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < h; k += blockDim.x) {
        double s = 0.0;
        int a = 0;  // k x mod n
        for (int x = 0; x < h; x++) {
            s = fma(sg[x], tw[a].x, s);
            a += k;
            if (a >= n) a -= n;
        }
        T[((long long)z * h + k) * hy + y] = s;
    }
}

__global__ void k_conv_table_y(const double *__restrict__ T, double *__restrict__ G, const double2 *__restrict__ tw,
                               int n, int h, int hx, int Z, double scale)
{
    extern __shared__ double sg[];
    const int z = blockIdx.x % Z, kx = blockIdx.x / Z;
    for (int y = threadIdx.x; y < h; y += blockDim.x)
        sg[y] = T[((long long)z * hx + kx) * h + y] * (y == 0 || 2 * y == n ? 1.0 : 2.0);
    __syncthreads();
    for (int k = threadIdx.x; k < h; k += blockDim.x) {
        double s = 0.0;
        int a = 0;
        for (int y = 0; y < h; y++) {
            s = fma(sg[y], tw[a].x, s);
            a += k;
            if (a >= n) a -= n;
        }
        G[((long long)kx * Z + z) * h + k] = s * scale;
    }
}

// ---- the passes with the columns in device memory [kx][z][y] -------------------
// Three launches a potential.  Up to about 200 cells a side they are bound by
// launch and barrier latency (4 us each); at 256 x 256 x 3 still by the latency of
// loads (8 to 11 warps an SM, issue 13 to 18 %, FP64 pipe 8 to 14 %, L2 6 %).
// Beyond, the column store's traffic grows with the cells (32 bytes a cell and
// pass).  Measured, whole
// potential, against the pair sum: 64 x 64 x 3 8.7 us (100 us), 256 x 256 x 3
// 18.7 us (2,056 us), 512 x 512 x 3 68 us (23.9 ms), 1024 x 1024 x 3 294 us
// (382 ms); rel-L2 against the FP64 sum 2.5e-8 at every size, the rounding of
// phi to FP32 (the compensated FP32 pair sum: 2e-7 .. 9e-7).  Columns are kept
// [kx][z][y]: the column pass streams 16 Y bytes, and the four row pairs of a
// row CTA write and read whole 128-byte lines of each column (the way back
// with consecutive threads on consecutive pairs: 22 to 18.7 us at 256).  The row
// pass reads rho: forming the divergence of the state in it saves a launch but
// gave each thread 48 to 96 loads, 76 us a step of 76 x 27 x 3 cells against 55.
template <class PL>
__global__ void __launch_bounds__(MAX_THREADS) k_conv_rows(ConvDev c, const float *__restrict__ rho,
                                                           double2 *__restrict__ store)
{
    extern __shared__ __align__(16) double2 cbuf[];
    pdl_begin();
    const int np = c.Z * ((c.Y + 1) >> 1), p0 = blockIdx.x * c.fb, cs = c.cs, X = c.X, Y = c.Y;
    rows_forward<row_pairs<PL>(MAX_THREADS, ROW_PAIRS)>(PL{}, c, cbuf, p0, min(c.fb, np - p0),
                                                        [=](int z, int y) {
                                                            const float *r = rho + ((long long)z * Y + y) * X;
                                                            return [=](int x, bool) { return r[x]; };
                                                        },
                                                        [=](int k) { return store + (long long)k * cs; });
}

template <class PL>
__global__ void __launch_bounds__(MAX_THREADS) k_conv_columns(ConvDev c, double2 *__restrict__ store)
{
    extern __shared__ __align__(16) double2 cbuf[];
    pdl_begin();
    const int k0 = blockIdx.x * c.cpg, cs = c.cs;
    columns(PL{}, c, cbuf, min(c.cpg, c.hx - k0), [=](int j) { return store + (long long)(k0 + j) * cs; },
            [=](int j) { return k0 + j; });
}

template <class PL>
__global__ void __launch_bounds__(MAX_THREADS) k_conv_back(ConvDev c, const double2 *__restrict__ store,
                                                           float *__restrict__ phi)
{
    extern __shared__ __align__(16) double2 cbuf[];
    pdl_begin();
    const int np = c.Z * ((c.Y + 1) >> 1), p0 = blockIdx.x * c.fb, cs = c.cs, X = c.X, Y = c.Y;
    rows_back<row_pairs<PL>(MAX_THREADS, ROW_PAIRS)>(PL{}, c, cbuf, p0, min(c.fb, np - p0),
                                                     [=](int k) { return store + (long long)k * cs; },
                                                     [=](int z, int y) {
                                                         float *r = phi + ((long long)z * Y + y) * X;
                                                         return [=](int x, float v) { r[x] = v; };
                                                     });
}

}  // namespace

namespace mmsconv {

// the shortest transform for m cells: at least 2 m - 1 long, so that no
// wrap-around reaches a cell
static bool fft_plan(int m, bool batch, int threads, int most, FftPlan &p, int *pairs)
{
    for (int id = 0; id < (batch ? NBATCH : NPLANS); id++) {
        auto take = [&](auto pl) {
            using PL = decltype(pl);
            p = FftPlan{id, PL::n, PL::stride, PL::mmax};
            *pairs = row_pairs<PL>(threads, most);
        };
        if (batch)
            with_batch_plan_host(id, take);
        else
            with_plan(id, take);
        if (p.n >= 2 * m - 1 && p.mmax <= threads) return true;
    }
    return false;
}

bool conv_layout(ConvDev &c, int X, int Y, int Z, bool batch, int threads, int pairs, size_t *smem)
{
    c = ConvDev{};
    int unused = 0;
    if (X < 1 || Y < 1 || Z < 1 || Z > ZMAX || !fft_plan(X, batch, threads, pairs, c.px, &c.fb) ||
        !fft_plan(Y, batch, threads, pairs, c.py, &unused))
        return false;
    c.X = X;
    c.Y = Y;
    c.Z = Z;
    c.hx = c.px.n / 2 + 1;
    c.hy = c.py.n / 2 + 1;
    c.ys = (Y + 1) / 2 * 2;
    c.cs = Z * c.ys;
    c.cpg = std::max(1, threads / (Z * c.py.mmax));
    *smem = std::max((size_t)c.fb * c.px.stride, (size_t)c.cpg * Z * c.py.stride) * sizeof(double2);
    return *smem <= SMEM_MAX;
}

size_t conv_table_bytes(const ConvDev &c)
{
    const size_t b = ((size_t)c.px.n + c.py.n) * sizeof(double2) + (size_t)c.hx * c.hy * c.Z * sizeof(double);
    return (b + 255) / 256 * 256;
}

size_t conv_table_scratch(const ConvDev &c) { return (size_t)c.hx * c.hy * c.Z * sizeof(double); }

int conv_build_tables(ConvDev &c, void *tab, double *scratch, double dx, double dy, double dz, cudaStream_t st,
                      int64_t *launches)
{
    double2 *tx = (double2 *)tab, *ty = tx + c.px.n;
    double *g = (double *)(ty + c.py.n);
    k_conv_twiddle<<<div_up(c.px.n, 128), 128, 0, st>>>(tx, c.px.n);
    k_conv_twiddle<<<div_up(c.py.n, 128), 128, 0, st>>>(ty, c.py.n);
    k_conv_table_x<<<c.hy * c.Z, 128, c.hx * sizeof(double), st>>>(scratch, tx, c.px.n, c.hx, c.hy, dx, dy, dz);
    k_conv_table_y<<<c.hx * c.Z, 128, c.hy * sizeof(double), st>>>(scratch, g, ty, c.py.n, c.hy, c.hx, c.Z,
                                                                   0.5 / ((double)c.px.n * c.py.n));
    MMS_CUDA_TRY(cudaGetLastError());
    *launches += 4;
    c.twx = tx;
    c.twy = ty;
    c.G = g;
    return MMS_OK;
}

}  // namespace mmsconv

struct ConvPlan {
    ConvDev g{};               // columns in device memory
    void *mem = nullptr;       // column store, then the tables
    double2 *store = nullptr;
    size_t bytes = 0;
};

// layout and memory of a grid's plan: column store (first the tables'
// scratch), tables; 0 bytes where there is none
static size_t plan_layout(const mms_grid &g, ConvDev &c, size_t *smem, size_t *first)
{
    if (!conv_layout(c, g.xdim, g.ydim, g.zdim, false, MAX_THREADS, ROW_PAIRS, smem)) return 0;
    c.cpg = 1;  // a CTA per column: the launch has few enough
    const size_t store = (size_t)c.hx * c.cs * sizeof(double2);
    *first = (std::max(store, conv_table_scratch(c)) + 255) / 256 * 256;
    return *first + conv_table_bytes(c);
}

size_t conv_plan_bytes(const mms_grid &g)
{
    ConvDev c;
    size_t smem = 0, first = 0;
    return plan_layout(g, c, &smem, &first);
}

// The convolution plan of a context's grid; *out stays NULL (and MMS_OK) where
// the pair sum serves the grid: more than ZMAX layers, rows or columns beyond
// the transforms' length (2,048 cells), no memory for the column store, or
// columns that a CTA cannot hold: all layers of one are transformed together,
// 16 bytes for each of Z padded transforms, in at most 200 KB.  Beyond 512 cells
// along y that means fewer layers: 7 to 768 cells, 5 to 1,024, 2 to 2,048 (along
// x rows have no such limit: lay the longer side there).
int conv_plan_create(mms_ctx *ctx, ConvPlan **out)
{
    *out = nullptr;
    ConvPlan pl;
    ConvDev &c = pl.g;
    size_t smem = 0, first = 0;
    pl.bytes = plan_layout(ctx->g, c, &smem, &first);
    if (!pl.bytes || ctx_alloc(ctx, (char **)&pl.mem, pl.bytes) != MMS_OK) return MMS_OK;
    pl.store = (double2 *)pl.mem;
    int st = conv_build_tables(c, (char *)pl.mem + first, (double *)pl.mem, ctx->g.dx, ctx->g.dy, ctx->g.dz,
                               ctx->stream, &ctx->launches);
    with_plan(pl.g.px.id, [&](auto p) {
        if (!st) st = allow_smem((const void *)k_conv_rows<decltype(p)>, smem);
        if (!st) st = allow_smem((const void *)k_conv_back<decltype(p)>, smem);
    });
    with_plan(pl.g.py.id, [&](auto p) {
        if (!st) st = allow_smem((const void *)k_conv_columns<decltype(p)>, smem);
    });
    if (st) {
        ctx_free(ctx, pl.mem);
        return st;
    }
    *out = new ConvPlan(pl);
    return MMS_OK;
}

void conv_plan_destroy(mms_ctx *ctx)
{
    if (!ctx->conv) return;
    ctx_free(ctx, ctx->conv->mem);
    delete ctx->conv;
    ctx->conv = nullptr;
}

int launch_potential_conv(mms_ctx *ctx, ConvPlan *pl, const float *rho, float *phi)
{
    const ConvDev &c = pl->g;
    const int pairs = c.Z * ((c.Y + 1) / 2);
    const unsigned tr = (c.fb * c.px.mmax + 31) / 32 * 32;
    const unsigned tc = std::min(MAX_THREADS, (c.Z * c.py.mmax + 31) / 32 * 32);
    const size_t sr = (size_t)c.fb * c.px.stride * sizeof(double2);
    const size_t sc = (size_t)c.cpg * c.Z * c.py.stride * sizeof(double2);
    cudaError_t e = cudaSuccess;
    with_plan(c.px.id, [&](auto p) {
        e = launch_k(k_conv_rows<decltype(p)>, dim3(div_up(pairs, c.fb)), dim3(tr), sr, ctx->stream, c, rho, pl->store);
    });
    MMS_CUDA_TRY(e);
    MMS_LAUNCH_CHECK(ctx);
    with_plan(c.py.id, [&](auto p) {
        e = launch_k(k_conv_columns<decltype(p)>, dim3(div_up(c.hx, c.cpg)), dim3(tc), sc, ctx->stream, c, pl->store);
    });
    MMS_CUDA_TRY(e);
    MMS_LAUNCH_CHECK(ctx);
    with_plan(c.px.id, [&](auto p) {
        e = launch_k(k_conv_back<decltype(p)>, dim3(div_up(pairs, c.fb)), dim3(tr), sr, ctx->stream, c,
                     (const double2 *)pl->store, phi);
    });
    MMS_CUDA_TRY(e);
    MMS_LAUNCH_CHECK(ctx);
    return MMS_OK;
}
