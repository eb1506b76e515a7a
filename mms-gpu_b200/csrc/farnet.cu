// Training of the learned far-field network (mms_farnet_*): forward pass,
// relative-L2 loss against far-field targets, adjoint passes, weight
// gradients on the tensor cores, Adam.
//
// The network (farnet.cuh) is the FMM's data flow with its own weights per
// level: encoder (P2M), down (M2M), interaction-list lateral (M2L), up (L2L),
// decoder (L2P); the exact near field is not part of it.  Activations are
// FP32, one [batch][box][NR] tensor per kind over the boxes of every level
// (levels 2..L, level-major, box row-major inside a level):
//   M   multipoles           Lf  final locals (M2L + L2L of the parent's)
//   dM  dloss/dM             dL  dloss/dLf
// Every forward and adjoint kernel gives each output element to one thread (no
// atomics: fixed summation order, reproducible bits, of the gradients too; the
// loss alone is added up over CTAs by FP64 atomics, so its last bits vary): the
// levels that do not depend on one another share a launch (the interaction lists
// of every level), the chains along the tree are a CTA per level-2 box that walks
// its levels.  The gradients of the translation tables are sums of outer products
// over boxes and samples with 320 wanted entries an operator, in FP32 registers
// (k_t_opgrad; within 5e-6 of the split-BF16 GEMMs they were); those of the
// encoder and the decoder, 192 x 24 with K = boxes x samples, are GEMMs: the
// operands are gathered into K-major BF16 hi/lo planes
// ([hi | lo | hi] against [hi | hi | lo], relative error ~2^-16 per product)
// and multiplied by the tcgen05 core (umma_gemm_bf16_splitk: the long K range
// split over CTAs, the partials summed in a fixed order).
//
// A gradient of 8 samples of 256 x 256 x 3 took 1,320 us with a thread per
// output everywhere, a launch per level and every table's gradient a gathered
// GEMM (a 58 MB operand for the leaf level's interaction lists): some 75
// launches, the largest 138, 130 and 128 us.  Now 278 us: 19 launches of 205 us
// (lists 2 x 22, k_t_opgrad 24, leaves 17, operands 17, GEMMs and their sums
// 39, chains 35), bound by latency with few warps an SM (the lists by shared-memory
// reads), and the results' way to the host.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>

#include "farnet.cuh"
#include "mms_internal.cuh"
#include "umma.cuh"

using bf16 = __nv_bfloat16;

// what the host reads of a gradient: the loss and the GEMM core's error word
struct FarnetResult {
    double loss;
    int err, pad;
};

struct mms_farnet {
    int X = 0, Y = 0, L = 0, nb = 0, batch = 0;
    long long N = 0;     // cells per sample (FN_Z * Y * X)
    long long nbox = 0;  // boxes of levels 2..L
    long long lev_off[FN_DEPTHS + 3] = {};
    long long *lev_dev = nullptr;
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // weights, gradient, Adam moments
    float *wt = nullptr;  // weights with transposed translation tables (of the last gradient)
    float *sc = nullptr;  // per-weight step scale (1 unless set)
    float *M = nullptr, *Lf = nullptr, *dM = nullptr, *dL = nullptr;
    float *dout = nullptr;
    double *lsum = nullptr;
    FarnetResult *res = nullptr;
    void *host = nullptr;        // pinned: a FarnetResult, then a gradient
    const int *err = nullptr;    // the GEMM core's error word (device)
    bf16 *ops = nullptr;   // GEMM operands of the encoder's and decoder's gradients
    float *Cp = nullptr;   // partial sums of the weight gradients
    size_t p_elems = 0;
    long long step = 0;
    size_t bytes = 0;
};

namespace {

struct NetK {
    int X, Y, L, nb, batch;
    long long N, nbox;
    long long lev[FN_DEPTHS + 3];
};

// o = (ox, oy) lies in the interaction list of the box at (tx, ty)
__device__ __forceinline__ bool in_list(int ox, int oy, int tx, int ty)
{
    const int px = tx & 1, py = ty & 1;
    return max(abs(ox), abs(oy)) >= 2 && ox >= px - 3 && ox <= px + 2 && oy >= py - 3 && oy <= py + 2;
}

// the translation tables with their blocks transposed, for the adjoints (which
// then read them input-major as the forward passes do)
__global__ void k_t_transpose(const float *__restrict__ w, float *__restrict__ wt, int nops)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nops * FN_OSZ) return;
    const int e = i % FN_OSZ;
    const bool odd = e >= FN_NE * FN_NE;
    const int n = odd ? FN_NO : FN_NE, ee = odd ? e - FN_NE * FN_NE : e;
    wt[fn_off_M2L(0) + i] = w[fn_off_M2L(0) + i - ee + (ee % n) * n + ee / n];
}

// n floats (a multiple of 4, 16-byte aligned) into shared memory, every copy in
// flight at once; stage_wait and a __syncthreads before they are read
__device__ __forceinline__ void stage(float *dst, const float *src, int n)
{
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) umma::cp_async16(umma::smem_u32(dst + i), src + i, true);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// out_k = sum_j T[j][k] x_j, T in shared memory, x a row of global memory
// that this launch may have written (16-byte aligned)
__device__ __forceinline__ float row_apply(const float *T, const float *x, int k)
{
    float acc = 0.f;
    if (k < FN_NE) {
#pragma unroll
        for (int v = 0; v < FN_NE / 4; v++) {
            const float4 a = reinterpret_cast<const float4 *>(x)[v];
            acc = fmaf(T[(4 * v) * FN_NE + k], a.x, acc);
            acc = fmaf(T[(4 * v + 1) * FN_NE + k], a.y, acc);
            acc = fmaf(T[(4 * v + 2) * FN_NE + k], a.z, acc);
            acc = fmaf(T[(4 * v + 3) * FN_NE + k], a.w, acc);
        }
    } else {
        const float *To = T + FN_NE * FN_NE + k - FN_NE;
#pragma unroll
        for (int v = 0; v < FN_NO / 4; v++) {
            const float4 a = reinterpret_cast<const float4 *>(x + FN_NE)[v];
            acc = fmaf(To[(4 * v) * FN_NO], a.x, acc);
            acc = fmaf(To[(4 * v + 1) * FN_NO], a.y, acc);
            acc = fmaf(To[(4 * v + 2) * FN_NO], a.z, acc);
            acc = fmaf(To[(4 * v + 3) * FN_NO], a.w, acc);
        }
    }
    return acc;
}

constexpr int TBOX = 32;            // leaf boxes per CTA in k_t_p2m
constexpr int TPITCH = FN_C + 4;    // floats per staged leaf box

// leaf box number i of nbatch nb^2 (sample-major): sample, box, its corner
__device__ __forceinline__ void leaf_of(const NetK &k, long long i, int &b, int &box, int &x0, int &y0)
{
    const int sh = k.L;  // nb = 1 << L boxes a side
    b = (int)(i >> (2 * sh));
    box = (int)i & ((1 << (2 * sh)) - 1);
    x0 = (box & (k.nb - 1)) * FN_S;
    y0 = (box >> sh) * FN_S;
}

// the cells of boxes i0 .. i0 + NBOX - 1 of a [batch][3][Y][X] array into
// [box][cell], zero off the grid (consecutive threads on consecutive cells of a
// row, then the next box)
template <int NBOX, int PITCH>
__device__ __forceinline__ void stage_boxes(float *q, const float *__restrict__ a, const NetK &k, long long i0,
                                            long long nbox)
{
    constexpr int U = 8;  // loads in flight
    for (int e0 = threadIdx.x; e0 < NBOX * FN_C; e0 += U * blockDim.x) {
        float v[U];
#pragma unroll
        for (int r = 0; r < U; r++) {
            const int e = e0 + r * blockDim.x, xx = e % FN_S, bl = e / FN_S % NBOX, row = e / (FN_S * NBOX);
            int b, box, x0, y0;
            leaf_of(k, min(i0 + bl, nbox - 1), b, box, x0, y0);
            const int x = x0 + xx, y = y0 + row % FN_S, z = row / FN_S;
            const bool ok = e < NBOX * FN_C && i0 + bl < nbox && x < k.X && y < k.Y;
            v[r] = ok ? __ldg(&a[(long long)b * k.N + ((long long)z * k.Y + y) * k.X + x]) : 0.f;
        }
#pragma unroll
        for (int r = 0; r < U; r++) {
            const int e = e0 + r * blockDim.x, xx = e % FN_S, bl = e / FN_S % NBOX, row = e / (FN_S * NBOX);
            if (e < NBOX * FN_C) q[bl * PITCH + row * FN_S + xx] = v[r];
        }
    }
}

// encoder: M[b][leaf][k] = sum_c W[c][k] u[b][cell(leaf, c)].  CTA = TBOX leaf
// boxes, staged with the weights; a thread sums one channel of four boxes.
__global__ void __launch_bounds__(8 * FN_NR) k_t_p2m(const float *__restrict__ u, const float *__restrict__ w,
                                                     float *__restrict__ M, NetK k)
{
    extern __shared__ __align__(16) float sm[];
    float *q = sm, *W = sm + TBOX * TPITCH;
    const long long nbox = (long long)k.batch * k.nb * k.nb, i0 = (long long)blockIdx.x * TBOX;
    stage(W, w + fn_off_W(), FN_C * FN_NR);
    stage_boxes<TBOX, TPITCH>(q, u, k, i0, nbox);
    stage_wait();
    __syncthreads();
    const int ch = threadIdx.x % FN_NR, g = threadIdx.x / FN_NR;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int c = 0; c < FN_C; c += 4) {
        const float w0 = W[c * FN_NR + ch], w1 = W[(c + 1) * FN_NR + ch], w2 = W[(c + 2) * FN_NR + ch],
                    w3 = W[(c + 3) * FN_NR + ch];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 v = *reinterpret_cast<const float4 *>(&q[(4 * g + i) * TPITCH + c]);
            acc[i] = fmaf(w0, v.x, acc[i]);
            acc[i] = fmaf(w1, v.y, acc[i]);
            acc[i] = fmaf(w2, v.z, acc[i]);
            acc[i] = fmaf(w3, v.w, acc[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (i0 + 4 * g + i >= nbox) break;
        int b, box, x0, y0;
        leaf_of(k, i0 + 4 * g + i, b, box, x0, y0);
        M[((long long)b * k.nbox + k.lev[k.L] + box) * FN_NR + ch] = acc[i];
    }
}

constexpr int CHAIN_THREADS = 256;
constexpr int CHAIN_LEVELS = FN_DEPTHS - 1;  // tables a chain holds: levels 2 .. L-1

// a chain's tables (of parent levels L-1 .. 2; [l - 2]) in flight at once
template <bool ADJ>
__device__ __forceinline__ void stage_chain(float *T, const float *w, const NetK &k, bool up)
{
    for (int l = 2; l < k.L; l++)
        stage(T + (l - 2) * 4 * FN_OSZ, w + (up ? fn_off_M2M(k.L - l) : fn_off_L2L(k.L - l)), 4 * FN_OSZ);
    stage_wait();
    __syncthreads();
}

// Chains from the leaves up, CTA = (sample, level-2 box) and all its boxes of
// levels L-1 .. 2: parent = sum of its four children through their operators.
// Forward: the multipoles, M2M.  ADJ: dL through the transposed L2L (w: the
// transposed tables).
template <bool ADJ>
__global__ void __launch_bounds__(CHAIN_THREADS) k_t_ascend(const float *__restrict__ w, float *A, NetK k)
{
    __shared__ __align__(16) float Ts[CHAIN_LEVELS * 4 * FN_OSZ];
    const int bx2 = blockIdx.x % 4, by2 = blockIdx.x / 4 % 4;
    float *Ab = A + (long long)(blockIdx.x / 16) * k.nbox * FN_NR;
    stage_chain<ADJ>(Ts, w, k, !ADJ);
    for (int l = k.L - 1; l >= 2; l--) {
        const float *T = Ts + (l - 2) * 4 * FN_OSZ;
        const int sh = l - 2, n = 1 << l;
        for (int e = threadIdx.x; e < FN_NR << (2 * sh); e += blockDim.x) {
            const int ch = e % FN_NR, p = e / FN_NR;
            const int px = (bx2 << sh) + (p & ((1 << sh) - 1)), py = (by2 << sh) + (p >> sh);
            float acc = 0.f;
#pragma unroll
            for (int c = 0; c < 4; c++)
                acc += row_apply(T + c * FN_OSZ,
                                 Ab + (k.lev[l + 1] + (long long)(2 * py + (c >> 1)) * 2 * n + 2 * px + (c & 1)) * FN_NR, ch);
            Ab[(k.lev[l] + (long long)py * n + px) * FN_NR + ch] = acc;
        }
        __syncthreads();
    }
}

// Chains from level 2 down, the same CTAs: each box adds its parent's row
// through its operator to what the interaction lists gave it.  Forward: the
// locals, L2L.  ADJ: dM through the transposed M2M.
template <bool ADJ>
__global__ void __launch_bounds__(CHAIN_THREADS) k_t_descend(const float *__restrict__ w, float *A, NetK k)
{
    __shared__ __align__(16) float Ts[CHAIN_LEVELS * 4 * FN_OSZ];
    const int bx2 = blockIdx.x % 4, by2 = blockIdx.x / 4 % 4;
    float *Ab = A + (long long)(blockIdx.x / 16) * k.nbox * FN_NR;
    stage_chain<ADJ>(Ts, w, k, ADJ);
    for (int l = 3; l <= k.L; l++) {
        const float *T = Ts + (l - 3) * 4 * FN_OSZ;
        const int sh = l - 2, n = 1 << l;
        for (int e = threadIdx.x; e < FN_NR << (2 * sh); e += blockDim.x) {
            const int ch = e % FN_NR, p = e / FN_NR;
            const int tx = (bx2 << sh) + (p & ((1 << sh) - 1)), ty = (by2 << sh) + (p >> sh);
            float *o = Ab + (k.lev[l] + (long long)ty * n + tx) * FN_NR + ch;
            const float own = *o;
            *o = own + row_apply(T + ((ty & 1) * 2 + (tx & 1)) * FN_OSZ,
                                 Ab + (k.lev[l - 1] + (long long)(ty >> 1) * (n >> 1) + (tx >> 1)) * FN_NR, ch);
        }
        __syncthreads();
    }
}

// the class's list offset number i
__device__ __forceinline__ void list_offset(int i, int px, int py, int &ox, int &oy)
{
    int at = 0;
    for (oy = py - 3; oy <= py + 2; oy++)
        for (ox = px - 3; ox <= px + 2; ox++)
            if (max(abs(ox), abs(oy)) >= 2 && at++ == i) return;
}

// two independent FMAs in one instruction, each rounded as fmaf
__device__ __forceinline__ void fma2(float2 &acc, float2 a, float2 b)
{
    unsigned long long &c = reinterpret_cast<unsigned long long &>(acc);
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(c)
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
}

// The interaction lists of every level in one launch.  CTA = 32 boxes of one
// level and parity class, lane = box, a warp a sixth of their channels (even 4 w
// .. 4 w + 3, or odd): per offset the CTA's 192 threads bring the 32 source rows
// into shared memory (a 16-byte piece each, two offsets ahead, two buffers) and
// every lane multiplies its row by the operator's, read as 16-byte broadcasts.
//   forward: out[t] = sum_o T[o] in[t - o], o in the list of t
//   ADJ:     out[s] = sum_o T[o]^T in[s + o], o in the list of s + o
// Bound by shared-memory reads (L1 pipe 70 %, issue 33 %).  8 x 256 x 256: 27 us
// with a third of the channels a warp and rows of its own, 34 us with two
// boxes a lane besides (half the operator reads, half the warps); 22 us as here.
constexpr int LAT_BOXES = 32, LAT_THREADS = 6 * 32;
constexpr int LAT_PITCH = FN_NR + 4;  // floats of a row in a buffer
constexpr size_t LAT_SMEM = (49 * FN_OSZ + 2 * LAT_BOXES * LAT_PITCH) * sizeof(float);
struct LatK {
    int cta[FN_DEPTHS + 3];     // first CTA of level l (finest level first), [1]: their number
    int groups[FN_DEPTHS + 3];  // groups per parity class
};

template <bool ADJ>
__global__ void __launch_bounds__(LAT_THREADS) k_t_lateral(const float *__restrict__ w, const float *__restrict__ in,
                                                           float *__restrict__ out, NetK k, LatK lk)
{
    extern __shared__ __align__(16) float Ts[];
    int l = k.L;
    while (l > 2 && (int)blockIdx.x >= lk.cta[l - 1]) l--;
    stage(Ts, w + fn_off_M2L(k.L - l), 49 * FN_OSZ);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = blockIdx.x - lk.cta[l];
    const int cls = grp / lk.groups[l], px = cls & 1, py = cls >> 1, n = 1 << l, sh = l - 1;  // n / 2 boxes a side
    const long long t0 = (long long)(grp % lk.groups[l]) * LAT_BOXES, nt = (long long)k.batch << (2 * sh);
    // box number i of the group, its level's first row; false where there is none
    auto box = [&](int i, int &tx, int &ty, long long &row0) {
        const long long ti = t0 + i;
        const int t = (int)ti & ((1 << (2 * sh)) - 1);
        tx = 2 * (t & ((1 << sh) - 1)) + px;
        ty = 2 * (t >> sh) + py;
        row0 = (ti < nt ? ti >> (2 * sh) : 0) * k.nbox + k.lev[l];
        return ti < nt;
    };
    // the class's 27 offsets, lane i the i-th; those of the adjoint's lists are
    // the other parity's
    int my_ox, my_oy;
    list_offset(min(lane, 26), ADJ ? 1 - px : px, ADJ ? 1 - py : py, my_ox, my_oy);
    float *buf = Ts + 49 * FN_OSZ;
    int hx, hy;  // the box whose source rows this thread loads a piece of
    long long h0;
    const bool hv = box(threadIdx.x / 6, hx, hy, h0);
    const int piece = 4 * (threadIdx.x % 6);
    float *mine = buf + threadIdx.x / 6 * LAT_PITCH + piece;
    auto fetch = [&](int i) {
        const int ox = __shfl_sync(0xffffffffu, my_ox, min(i, 26)), oy = __shfl_sync(0xffffffffu, my_oy, min(i, 26));
        const int sx = ADJ ? hx + ox : hx - ox, sy = ADJ ? hy + oy : hy - oy;
        const bool ok = hv && sx >= 0 && sy >= 0 && sx < n && sy < n;
        const float4 q = __ldg(reinterpret_cast<const float4 *>(in + (h0 + (ok ? (sy << l) + sx : 0)) * FN_NR + piece));
        return ok ? q : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    // the lane's row times this warp's channels of operator o
    auto times = [&](auto odd, const float *row, int o) {
        constexpr int J = decltype(odd)::value ? FN_NO : FN_NE;
        const float *T = Ts + o * FN_OSZ + (J == FN_NO ? FN_NE * FN_NE + 4 * (warp - 4) : 4 * warp);
        row += J == FN_NO ? FN_NE : 0;
        float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
        for (int v = 0; v < J / 4; v++) {
            const float4 q = *reinterpret_cast<const float4 *>(row + 4 * v);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 a = *reinterpret_cast<const float4 *>(T + (4 * v + j) * J);
                const float b = j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : q.w;
                fma2(s0, make_float2(a.x, a.y), make_float2(b, b));
                fma2(s1, make_float2(a.z, a.w), make_float2(b, b));
            }
        }
        acc[0] += s0.x;
        acc[1] += s0.y;
        acc[2] += s1.x;
        acc[3] += s1.y;
    };
    float4 x0 = fetch(0), x1 = fetch(1);
    stage_wait();
    auto step = [&](float4 &x, int i) {
        const int at = (i & 1) * LAT_BOXES * LAT_PITCH;
        *reinterpret_cast<float4 *>(mine + at) = x;
        x = fetch(i + 2);
        const int ox = __shfl_sync(0xffffffffu, my_ox, i), oy = __shfl_sync(0xffffffffu, my_oy, i);
        __syncthreads();  // (the other buffer is free again: its readers came here after they were done)
        const float *row = buf + at + lane * LAT_PITCH;
        const int o = (oy + 3) * 7 + ox + 3;
        if (warp >= 4)
            times(std::true_type{}, row, o);
        else
            times(std::false_type{}, row, o);
    };
#pragma unroll 1
    for (int i = 0; i < 26; i += 2) {
        step(x0, i);
        step(x1, i + 1);
    }
    step(x0, 26);
    int tx, ty;
    long long row0;
    if (!box(lane, tx, ty, row0)) return;
    *reinterpret_cast<float4 *>(out + (row0 + (ty << l) + tx) * FN_NR + 4 * warp) = make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// decoder: out[b][cell] = sum_k V[k][c] Lf_L[b][leaf][k].  CTA = LEAF_BOXES leaf
// boxes, thread = cell c with its 24 weights in registers.  LOSS: the loss
// sums, the output adjoint dout = 2 (out - far) / (nrm_b batch) in place of
// out, and its own adjoint dL_L[b][leaf][k] = sum_c V[k][c] dout.
constexpr int LEAF_BOXES = 16;
constexpr int VPITCH = FN_C + 4;
template <bool LOSS>
__global__ void __launch_bounds__(FN_C) k_t_leaf(const float *__restrict__ w, const float *__restrict__ Lf,
                                                 float *__restrict__ out, const float *__restrict__ far,
                                                 const float *__restrict__ nrm, double *__restrict__ lsum,
                                                 float *__restrict__ dL, NetK k, int nbatch)
{
    __shared__ __align__(16) float V[FN_NR * VPITCH];
    __shared__ __align__(16) float rows[LEAF_BOXES * FN_NR];
    __shared__ __align__(16) float d[LOSS ? LEAF_BOXES * VPITCH : 4];
    __shared__ double red[FN_C / 32];
    const long long i0 = (long long)blockIdx.x * LEAF_BOXES;  // 16 divides the boxes of a sample
    const int c = threadIdx.x;
    float v[FN_NR];
#pragma unroll
    for (int ch = 0; ch < FN_NR; ch++) {
        v[ch] = __ldg(&w[fn_off_V() + ch * FN_C + c]);
        if (LOSS) V[ch * VPITCH + c] = v[ch];
    }
    for (int e = threadIdx.x; e < LEAF_BOXES * FN_NR; e += blockDim.x) {
        int b, box, x0, y0;
        leaf_of(k, i0 + e / FN_NR, b, box, x0, y0);
        rows[e] = Lf[((long long)b * k.nbox + k.lev[k.L] + box) * FN_NR + e % FN_NR];
    }
    __syncthreads();
    double r2 = 0.0;
#pragma unroll 8
    for (int i = 0; i < LEAF_BOXES; i++) {
        int b, box, x0, y0;
        leaf_of(k, i0 + i, b, box, x0, y0);
        const int x = x0 + c % FN_S, y = y0 + c / FN_S % FN_S, z = c / (FN_S * FN_S);
        const bool ok = x < k.X && y < k.Y;
        const long long cell = (long long)b * k.N + ((long long)z * k.Y + y) * k.X + x;
        float acc = 0.f;
#pragma unroll
        for (int ch = 0; ch < FN_NR; ch++) acc = fmaf(v[ch], rows[i * FN_NR + ch], acc);
        if (!LOSS) {
            if (ok) out[cell] = acc;
            continue;
        }
        float dv = 0.f;
        if (ok) {
            const float r = acc - far[cell];
            dv = 2.f * r / (nrm[b] * (float)nbatch);
            out[cell] = dv;
            r2 += (double)r * r;
        }
        d[i * VPITCH + c] = dv;
    }
    if (LOSS) {  // a CTA's boxes are of one sample (16 boxes or more each)
        for (int o = 16; o > 0; o >>= 1) r2 += __shfl_down_sync(0xffffffffu, r2, o);
        if ((c & 31) == 0) red[c >> 5] = r2;
        __syncthreads();
        if (c == 0) {
            double sum = 0.0;
            for (int q = 0; q < FN_C / 32; q++) sum += red[q];
            int b, box, x0, y0;
            leaf_of(k, i0, b, box, x0, y0);
            atomicAdd(&lsum[b], sum);
        }
    }
    if (!LOSS) return;
    // thread = (boxes i and i + 8, channel), the cells in order
    constexpr int H = FN_C / FN_NR, NB = LEAF_BOXES / H;
    const int i = c / FN_NR, ch = c % FN_NR;
    float acc[NB];
#pragma unroll
    for (int h = 0; h < NB; h++) acc[h] = 0.f;
#pragma unroll 4
    for (int q = 0; q < FN_C; q += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(&V[ch * VPITCH + q]);
#pragma unroll
        for (int h = 0; h < NB; h++) {
            const float4 e = *reinterpret_cast<const float4 *>(&d[(i + h * H) * VPITCH + q]);
            acc[h] = fmaf(a.x, e.x, acc[h]);
            acc[h] = fmaf(a.y, e.y, acc[h]);
            acc[h] = fmaf(a.z, e.z, acc[h]);
            acc[h] = fmaf(a.w, e.w, acc[h]);
        }
    }
#pragma unroll
    for (int h = 0; h < NB; h++) {
        int b, box, x0, y0;
        leaf_of(k, i0 + i + h * H, b, box, x0, y0);  // (16 boxes or more a sample: all exist)
        dL[((long long)b * k.nbox + k.lev[k.L] + box) * FN_NR + ch] = acc[h];
    }
}

// ---- weight gradients ---------------------------------------------------------
// Translation tables: g[op][j][k] = sum over rows of A[j] B[k], 20 tiles of 4 x
// 4 entries an operator (16 even, 4 odd), a thread per tile with its sums in
// registers, a CTA per chunk of rows; k_t_opsum adds the chunks in order and
// k_t_opscatter the classes (and the sub-rows).
//   M2L  level l, parity class: rows = its boxes t; op = the class's 27 offsets
//        A = M_l[t - o] (0 off the level), B = dL_l[t]
//   M2M  rows = parents p at level l; op = child c: A = M_{l+1}[c], B = dM_l[p]
//   L2L  the same rows; A = Lf_l[p], B = dL_{l+1}[c]
constexpr int OP_TILES = 20, OP_THREADS = 544;  // 27 x 20 tiles (540), or 6 rows at a time x 4 x 20 (480)
constexpr int OP_PART = OP_THREADS * 16;        // floats a chunk leaves
constexpr int OP_SUB = OP_THREADS / (4 * OP_TILES);
constexpr int OP_MAX_CHUNKS = 24;               // per class or family and level
struct OpK {
    // first item and chunks of M2L level l (4 classes), of M2M and of L2L with parents at level l
    int m2l[FN_DEPTHS + 3], m2l_ch[FN_DEPTHS + 3];
    int m2m[FN_DEPTHS + 3], l2l[FN_DEPTHS + 3], par_ch[FN_DEPTHS + 3];
    int items;
};

__device__ __forceinline__ void tile_of(int tile, int &j0, int &k0)
{
    const bool odd = tile >= 16;
    j0 = odd ? FN_NE + (tile - 16) / 2 * 4 : tile / 4 * 4;
    k0 = odd ? FN_NE + (tile - 16) % 2 * 4 : tile % 4 * 4;
}

__device__ __forceinline__ void outer(float (&acc)[16], const float4 a, const float4 b)
{
    const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[4 * i + j] = fmaf(x[i], y[j], acc[4 * i + j]);
}

__global__ void __launch_bounds__(OP_THREADS) k_t_opgrad(const float *__restrict__ M, const float *__restrict__ Lf,
                                                         const float *__restrict__ dM, const float *__restrict__ dL,
                                                         float *__restrict__ part, NetK k, OpK ok)
{
    const int item = blockIdx.x, t = threadIdx.x;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; i++) acc[i] = 0.f;
    int l = k.L;
    if (item < ok.m2m[2]) {  // M2L, finest level first
        while (l > 2 && item >= ok.m2l[l - 1]) l--;
        const int cls = (item - ok.m2l[l]) / ok.m2l_ch[l], chunk = (item - ok.m2l[l]) % ok.m2l_ch[l];
        const int px = cls & 1, py = cls >> 1, n = 1 << l, nh = n >> 1, sh = l - 1;
        const int lines = k.batch << sh, per = (lines + ok.m2l_ch[l] - 1) / ok.m2l_ch[l];  // lines of nh boxes
        if (t < 27 * OP_TILES) {
            int ox, oy, j0, k0;
            list_offset(t / OP_TILES, px, py, ox, oy);
            tile_of(t % OP_TILES, j0, k0);
            // boxes x = 2 q + px of a line whose source is on the level
            const int q0 = max(0, (ox - px + 1) >> 1), q1 = min(nh, (n + ox - px + 1) >> 1);
            const int r1 = min(lines, (chunk + 1) * per);
            for (int r = chunk * per; r < r1; r++) {
                const int b = r >> sh, ty = 2 * (r & (nh - 1)) + py, sy = ty - oy;
                if (sy < 0 || sy >= n) continue;
                const long long row0 = (long long)b * k.nbox + k.lev[l];
                const float *A = M + (row0 + (sy << l) + px - ox) * FN_NR + j0;
                const float *D = dL + (row0 + (ty << l) + px) * FN_NR + k0;
#pragma unroll 8
                for (int q = q0; q < q1; q++)
                    outer(acc, __ldg(reinterpret_cast<const float4 *>(A + q * 2 * FN_NR)),
                          __ldg(reinterpret_cast<const float4 *>(D + q * 2 * FN_NR)));
            }
        }
    } else {
        const bool up = item < ok.l2l[2];  // M2M, then L2L, coarsest parents first
        const int *first = up ? ok.m2m : ok.l2l;
        l = 2;
        while (l < k.L - 1 && item >= first[l + 1]) l++;
        const int chunk = item - first[l], n = 1 << l, lines = k.batch << l;
        const int per = (lines + ok.par_ch[l] - 1) / ok.par_ch[l];
        const int sub = t / (4 * OP_TILES), c = t / OP_TILES % 4;
        if (sub < OP_SUB) {
            int j0, k0;
            tile_of(t % OP_TILES, j0, k0);
            const int r1 = min(lines, (chunk + 1) * per);
            for (int r = chunk * per + sub; r < r1; r += OP_SUB) {
                const int b = r >> l, y = r & (n - 1);
                const long long base = (long long)b * k.nbox;
                const long long prow = (base + k.lev[l] + (y << l)) * FN_NR;
                const long long crow = (base + k.lev[l + 1] + ((2 * y + (c >> 1)) << (l + 1)) + (c & 1)) * FN_NR;
                const float *A = up ? M + crow + j0 : Lf + prow + j0, *D = up ? dM + prow + k0 : dL + crow + k0;
                const int sa = up ? 2 * FN_NR : FN_NR, sd = up ? FN_NR : 2 * FN_NR;
#pragma unroll 4
                for (int x = 0; x < n; x++)
                    outer(acc, __ldg(reinterpret_cast<const float4 *>(A + x * sa)),
                          __ldg(reinterpret_cast<const float4 *>(D + x * sd)));
            }
        }
    }
    float4 *o = reinterpret_cast<float4 *>(part + (long long)item * OP_PART + t * 16);
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
}

// the chunks of every (level, class) and (family, level), in order, into the
// first one's place: blockIdx.y = M2L of level 2 + y / 4, class y % 4, then M2M
// and L2L of parent levels 2, 3, ..
__global__ void k_t_opsum(float *__restrict__ part, NetK k, OpK ok)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, nm = 4 * (k.L - 1), y = blockIdx.y;
    if (i >= OP_PART / 4) return;
    int first, n;
    if (y < nm) {
        const int l = 2 + y / 4;
        n = ok.m2l_ch[l];
        first = ok.m2l[l] + y % 4 * n;
    } else {
        const int l = 2 + (y - nm) / 2;
        n = ok.par_ch[l];
        first = (y - nm) % 2 ? ok.l2l[l] : ok.m2m[l];
    }
    float4 *p = reinterpret_cast<float4 *>(part + (long long)first * OP_PART) + i;
    float4 s = p[0];
#pragma unroll 8
    for (int c = 1; c < n; c++) {
        const float4 v = p[(long long)c * (OP_PART / 4)];
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    }
    p[0] = s;
}

// those sums into the gradient vector: a thread per entry of the levels' M2L
// (49 slots, the near ones stay zero), M2M and L2L (4 children) tables
__global__ void k_t_opscatter(const float *__restrict__ part, float *__restrict__ g, NetK k, OpK ok)
{
    const int per_level = (49 + 4 + 4) * FN_OSZ;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int l = 2 + i / per_level;
    if (l > k.L) return;
    const int op = i % per_level / FN_OSZ, e = i % FN_OSZ;
    const bool odd = e >= FN_NE * FN_NE;
    const int ee = odd ? e - FN_NE * FN_NE : e, n = odd ? FN_NO : FN_NE, j = ee / n, q = ee % n;
    const int at = ((odd ? 16 + j / 4 * 2 : j / 4 * 4) + q / 4) * 16 + j % 4 * 4 + q % 4;  // tile, entry
    float s = 0.f;
    if (op < 49) {
        const int ox = op % 7 - 3, oy = op / 7 - 3;
        for (int cls = 0; cls < 4; cls++) {
            const int px = cls & 1, py = cls >> 1;
            if (!in_list(ox, oy, px, py)) continue;
            // its number in the class's list: the offsets before it, less the near ones
            const int rows = oy - (py - 3), cols = ox - (px - 3);
            const int near = 3 * max(0, min(3, oy + 1)) + (abs(oy) < 2 ? max(0, min(3, ox + 1)) : 0);
            s += part[(long long)(ok.m2l[l] + cls * ok.m2l_ch[l]) * OP_PART + (6 * rows + cols - near) * OP_TILES * 16 + at];
        }
        g[fn_off_M2L(k.L - l) + op * FN_OSZ + e] = s;
        return;
    }
    if (l == k.L) return;
    const int c = (op - 49) % 4;
    const bool up = op - 49 < 4;
    const float *p = part + (long long)(up ? ok.m2m[l] : ok.l2l[l]) * OP_PART + c * OP_TILES * 16 + at;
#pragma unroll
    for (int sub = 0; sub < OP_SUB; sub++) s += p[sub * 4 * OP_TILES * 16];
    g[(up ? fn_off_M2M(k.L - l) : fn_off_L2L(k.L - l)) + c * FN_OSZ + e] = s;
}

// The GEMMs' operands: W gradient [C][NR] = u dM_L^T, V gradient [NR][C] = Lf_L
// dout^T over the leaf boxes of all samples (K).  K-major planes of Kp elements
// a feature, side A [hi | lo | hi], side B [hi | hi | lo], zero beyond the
// boxes.  CTA = OBOX boxes of one pair, transposed through shared memory.
struct Operands {
    bf16 *u, *dM, *Lf, *dout;  // [C], [NR], [NR], [C] features
};

constexpr int OBOX = 64, OPITCH = FN_C + 1;  // read by feature: odd
constexpr size_t OPERANDS_SMEM = OBOX * (OPITCH + FN_NR + 1) * sizeof(float);

__global__ void __launch_bounds__(512) k_t_operands(const float *__restrict__ u, const float *__restrict__ dout,
                                                    const float *__restrict__ dM, const float *__restrict__ Lf,
                                                    Operands op, long long Kp, NetK k)
{
    extern __shared__ __align__(16) float sm[];
    float *q = sm, *rw = sm + OBOX * OPITCH;
    const long long nbox = (long long)k.batch * k.nb * k.nb, i0 = (long long)blockIdx.x * OBOX;
    const bool W = blockIdx.y == 0;  // u and dM, or dout and Lf
    stage_boxes<OBOX, OPITCH>(q, W ? u : dout, k, i0, nbox);
    const float *R = W ? dM : Lf;
    for (int e = threadIdx.x; e < OBOX * FN_NR; e += blockDim.x) {
        const int i = e / FN_NR, ch = e % FN_NR;
        int b, box, x0, y0;
        leaf_of(k, min(i0 + i, nbox - 1), b, box, x0, y0);
        const float v = __ldg(&R[((long long)b * k.nbox + k.lev[k.L] + box) * FN_NR + ch]);
        rw[i * (FN_NR + 1) + ch] = i0 + i < nbox ? v : 0.f;
    }
    __syncthreads();
    // a lane writes boxes 2 lane and 2 lane + 1 of a feature (Kp and i0 are even)
    const int lane = threadIdx.x & 31;
    if (i0 + 2 * lane >= Kp) return;
    for (int f = threadIdx.x >> 5; f < FN_C + FN_NR; f += blockDim.x >> 5) {
        const bool cell = f < FN_C;
        const float *src = cell ? q + 2 * lane * OPITCH + f : rw + 2 * lane * (FN_NR + 1) + f - FN_C;
        const float v0 = src[0], v1 = src[cell ? OPITCH : FN_NR + 1];
        const __nv_bfloat162 hi = __floats2bfloat162_rn(v0, v1);
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v0 - __low2float(hi), v1 - __high2float(hi));
        bf16 *row = (W ? (cell ? op.u : op.dM) : (cell ? op.dout : op.Lf)) + (long long)(cell ? f : f - FN_C) * 3 * Kp +
                    i0 + 2 * lane;
        const bool sideA = cell == W;  // u and Lf
        *reinterpret_cast<__nv_bfloat162 *>(row) = hi;
        *reinterpret_cast<__nv_bfloat162 *>(row + Kp) = sideA ? lo : hi;
        *reinterpret_cast<__nv_bfloat162 *>(row + 2 * Kp) = sideA ? hi : lo;
    }
}

__global__ void k_t_result(const double *__restrict__ lsum, const float *__restrict__ nrm, int nbatch,
                           const int *__restrict__ err, FarnetResult *__restrict__ r)
{
    double L = 0;
    for (int b = 0; b < nbatch; b++) L += lsum[b] / nrm[b];
    r->loss = L / nbatch;
    r->err = *err;
}

// Adam with a per-weight step scale: a weight moves by lr * sc_i per unit of
// normalised gradient, so tables whose entries span many orders of magnitude
// take relative steps
__global__ void k_t_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                         float *__restrict__ v, const float *__restrict__ sc, long long n, float lr, float b1,
                         float b2, float eps, float c1, float c2)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * sc[i] * (mi / c1) / (sqrtf(vi / c2) + eps);
}

__global__ void k_t_fill(float *__restrict__ a, long long n, float v)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = v;
}

NetK netk(const mms_farnet *n, int nbatch)
{
    NetK k;
    k.X = n->X;
    k.Y = n->Y;
    k.L = n->L;
    k.nb = n->nb;
    k.batch = nbatch;
    k.N = n->N;
    k.nbox = n->nbox;
    for (int i = 0; i < FN_DEPTHS + 3; i++) k.lev[i] = n->lev_off[i];
    return k;
}

constexpr int TB = 256;
inline unsigned nblk(long long n) { return (unsigned)((n + TB - 1) / TB); }

LatK latk(const mms_farnet *n, int nbatch)
{
    LatK k{};
    int at = 0;
    for (int l = n->L; l >= 2; l--) {
        k.cta[l] = at;
        k.groups[l] = (int)div_up((long long)nbatch << (2 * (l - 1)), LAT_BOXES);
        at += 4 * k.groups[l];
    }
    k.cta[1] = at;
    return k;
}

OpK opk(const mms_farnet *n, int nbatch)
{
    OpK k{};
    int at = 0;
    // 32 boxes a thread or more, whole lines of a level; from 24 chunks on (768
    // boxes of a class) the chunks get longer with the batch: 8 x 256 x 256 85
    // boxes, an FP32 sum of as many products
    auto chunks = [](long long boxes, long long lines) {
        return (int)std::max(1LL, std::min({(long long)OP_MAX_CHUNKS, boxes / 32, lines}));
    };
    for (int l = n->L; l >= 2; l--) {
        k.m2l[l] = at;
        k.m2l_ch[l] = chunks((long long)nbatch << (2 * (l - 1)), (long long)nbatch << (l - 1));
        at += 4 * k.m2l_ch[l];
    }
    for (int l = 2; l < n->L; l++)
        k.par_ch[l] = chunks(((long long)nbatch << (2 * l)) / OP_SUB, ((long long)nbatch << l) / OP_SUB);
    k.m2m[2] = at;
    for (int l = 2; l < n->L; l++) {
        k.m2m[l] = at;
        at += k.par_ch[l];
    }
    k.l2l[2] = at;
    for (int l = 2; l < n->L; l++) {
        k.l2l[l] = at;
        at += k.par_ch[l];
    }
    k.items = at;
    return k;
}

// the most chunks any batch of this network leaves
int op_items_max(int L) { return (L - 1) * 4 * OP_MAX_CHUNKS + 2 * std::max(0, L - 2) * OP_MAX_CHUNKS; }

// multipoles and final locals of nbatch samples
int forward(mms_farnet *n, const float *u, int nbatch)
{
    const NetK k = netk(n, nbatch);
    const LatK lk = latk(n, nbatch);
    cudaStream_t st = 0;
    const long long nl = (long long)n->nb * n->nb;
    const size_t smem = (TBOX * TPITCH + FN_C * FN_NR) * sizeof(float);
    k_t_p2m<<<div_up(nbatch * nl, TBOX), 8 * FN_NR, smem, st>>>(u, n->w, n->M, k);
    if (n->L > 2) k_t_ascend<false><<<16 * nbatch, CHAIN_THREADS, 0, st>>>(n->w, n->M, k);
    k_t_lateral<false><<<lk.cta[1], LAT_THREADS, LAT_SMEM, st>>>(n->w, n->M, n->Lf, k, lk);
    if (n->L > 2) k_t_descend<false><<<16 * nbatch, CHAIN_THREADS, 0, st>>>(n->w, n->Lf, k);
    MMS_CUDA_TRY(cudaGetLastError());
    return MMS_OK;
}

int gemm_gradient(mms_farnet *n, const bf16 *A, const bf16 *B, int fa, int fb, int K3, float *g)
{
    const int bn = fb <= 64 ? 64 : 128;
    int splits = 1, kchunk = K3;
    MMS_TRY(umma_gemm_bf16_splitk_plan(fa, fb, K3, bn, &splits, &kchunk));
    if ((size_t)splits * fa * fb > n->p_elems) {
        mms_set_error("farnet: split-K partial buffer too small");
        return MMS_ERR_ARG;
    }
    return umma_gemm_bf16_splitk(A, K3, B, K3, g, n->Cp, fa, fb, K3, bn, splits, kchunk, 0);
}

// Loss (host value) and the gradient into n->g, and into `grad` when it is
// given.  The results come through the network's pinned buffer with one
// synchronisation (pageable copies of each, waited for one by one, took about
// 60 us of a call).
int gradient(mms_farnet *n, const float *u, const float *far, const float *nrm2, int nbatch, double *loss, float *grad)
{
    MMS_TRY(forward(n, u, nbatch));
    const NetK k = netk(n, nbatch);
    const LatK lk = latk(n, nbatch);
    const OpK ok = opk(n, nbatch);
    const long long nl = (long long)n->nb * n->nb, rows = nbatch * nl, Kp = (rows + 7) / 8 * 8;
    if ((size_t)ok.items * OP_PART > n->p_elems) {
        mms_set_error("farnet: gradient partial buffer too small");
        return MMS_ERR_ARG;
    }
    MMS_CUDA_TRY(cudaMemsetAsync(n->lsum, 0, (size_t)nbatch * sizeof(double), 0));
    MMS_CUDA_TRY(cudaMemsetAsync(n->g, 0, (size_t)fn_num_params() * sizeof(float), 0));
    k_t_leaf<true><<<div_up(rows, LEAF_BOXES), FN_C>>>(n->w, n->Lf, n->dout, far, nrm2, n->lsum, n->dL, k, nbatch);
    const int nops = (int)((fn_num_params() - fn_off_M2L(0)) / FN_OSZ);
    k_t_transpose<<<nblk((long long)nops * FN_OSZ), TB>>>(n->w, n->wt, nops);
    if (n->L > 2) k_t_ascend<true><<<16 * nbatch, CHAIN_THREADS>>>(n->wt, n->dL, k);
    k_t_lateral<true><<<lk.cta[1], LAT_THREADS, LAT_SMEM>>>(n->wt, n->dL, n->dM, k, lk);
    if (n->L > 2) k_t_descend<true><<<16 * nbatch, CHAIN_THREADS>>>(n->wt, n->dM, k);
    k_t_opgrad<<<ok.items, OP_THREADS>>>(n->M, n->Lf, n->dM, n->dL, n->Cp, k, ok);
    k_t_opsum<<<dim3(nblk(OP_PART / 4), 4 * (n->L - 1) + 2 * (n->L - 2)), TB>>>(n->Cp, k, ok);
    k_t_opscatter<<<nblk((long long)(n->L - 1) * 57 * FN_OSZ), TB>>>(n->Cp, n->g, k, ok);
    Operands op;
    op.u = n->ops;
    op.dM = op.u + (size_t)FN_C * 3 * Kp;
    op.Lf = op.dM + (size_t)FN_NR * 3 * Kp;
    op.dout = op.Lf + (size_t)FN_NR * 3 * Kp;
    k_t_operands<<<dim3(div_up(Kp, OBOX), 2), 512, OPERANDS_SMEM>>>(u, n->dout, n->dM, n->Lf, op, Kp, k);
    MMS_CUDA_TRY(cudaGetLastError());
    MMS_TRY(gemm_gradient(n, op.u, op.dM, FN_C, FN_NR, (int)(3 * Kp), n->g + fn_off_W()));
    MMS_TRY(gemm_gradient(n, op.Lf, op.dout, FN_NR, FN_C, (int)(3 * Kp), n->g + fn_off_V()));
    k_t_result<<<1, 1>>>(n->lsum, nrm2, nbatch, n->err, n->res);
    MMS_CUDA_TRY(cudaGetLastError());
    const size_t gbytes = (size_t)fn_num_params() * sizeof(float);
    FarnetResult *hr = (FarnetResult *)n->host;
    float *hg = (float *)(hr + 1);
    MMS_CUDA_TRY(cudaMemcpyAsync(hr, n->res, sizeof(FarnetResult), cudaMemcpyDeviceToHost, 0));
    if (grad) MMS_CUDA_TRY(cudaMemcpyAsync(hg, n->g, gbytes, cudaMemcpyDeviceToHost, 0));
    MMS_CUDA_TRY(cudaStreamSynchronize(0));
    if (hr->err) {
        // (the word is the device's: another caller may have read and cleared it since)
        MMS_TRY(umma_check_error());
        mms_set_error("farnet: an mbarrier wait of a tensor-core GEMM timed out");
        return MMS_ERR_CUDA;
    }
    if (loss) *loss = hr->loss;
    if (grad) memcpy(grad, hg, gbytes);
    return MMS_OK;
}

int check_batch(const mms_farnet *n, int nbatch)
{
    if (!n || nbatch < 1 || nbatch > n->batch) {
        mms_set_error("farnet: bad network or batch size %d", nbatch);
        return MMS_ERR_ARG;
    }
    return MMS_OK;
}

}  // namespace

extern "C" {

long long mms_farnet_num_params(void) { return fn_num_params(); }

long long mms_surrogate_num_params(int width)
{
    if (width == FnTrain::NR) return FnTrain::num_params();
    if (width == FnWide::NR) return FnWide::num_params();
    return 0;
}

int mms_farnet_create(int xdim, int ydim, int batch, mms_farnet **out)
{
    if (!out || xdim < 1 || ydim < 1 || batch < 1) {
        mms_set_error("mms_farnet_create: bad argument");
        return MMS_ERR_ARG;
    }
    *out = nullptr;
    const int nleaf = std::max(1, (std::max(xdim, ydim) + FN_S - 1) / FN_S);
    int L = 0;
    while ((1 << L) < nleaf) L++;
    if (L < 2 || L > FN_DEPTHS + 1) {
        mms_set_error("mms_farnet_create: a %d x %d grid has %d quadtree levels; the network needs 2..%d", xdim, ydim,
                      L, FN_DEPTHS + 1);
        return MMS_ERR_ARG;
    }
    mms_farnet *n = new mms_farnet();
    n->X = xdim;
    n->Y = ydim;
    n->L = L;
    n->nb = 1 << L;
    n->batch = batch;
    n->N = (long long)FN_Z * xdim * ydim;
    long long tot = 0;
    for (int l = 2; l <= L; l++) {
        n->lev_off[l] = tot;
        tot += 1LL << (2 * l);
    }
    n->lev_off[L + 1] = tot;
    n->nbox = tot;
    const long long P = fn_num_params();
    const size_t act = (size_t)batch * tot * FN_NR;
    const long long Kp = ((long long)batch * n->nb * n->nb + 7) / 8 * 8;
    const size_t ops = (size_t)2 * (FN_C + FN_NR) * 3 * Kp;
    // partial sums: the operators' chunks, or up to one split per SM of a 192 x 24 gradient
    n->p_elems = std::max((size_t)op_items_max(L) * OP_PART, (size_t)FN_C * FN_NR * 148);
    struct {
        void **p;
        size_t bytes;
    } a[] = {{(void **)&n->w, P * sizeof(float)},
             {(void **)&n->wt, P * sizeof(float)},
             {(void **)&n->sc, P * sizeof(float)},
             {(void **)&n->g, P * sizeof(float)},
             {(void **)&n->m, P * sizeof(float)},
             {(void **)&n->v, P * sizeof(float)},
             {(void **)&n->M, act * sizeof(float)},
             {(void **)&n->Lf, act * sizeof(float)},
             {(void **)&n->dM, act * sizeof(float)},
             {(void **)&n->dL, act * sizeof(float)},
             {(void **)&n->dout, (size_t)batch * n->N * sizeof(float)},
             {(void **)&n->lsum, (size_t)batch * sizeof(double)},
             {(void **)&n->res, sizeof(FarnetResult)},
             {(void **)&n->ops, ops * sizeof(bf16)},
             {(void **)&n->Cp, n->p_elems * sizeof(float)},
             {(void **)&n->lev_dev, (FN_DEPTHS + 3) * sizeof(long long)}};
    for (auto &e : a) {
        if (cudaMalloc(e.p, e.bytes) != cudaSuccess) {
            mms_farnet_destroy(n);
            mms_set_error("mms_farnet_create: device allocation of %zu bytes failed", e.bytes);
            return MMS_ERR_NOMEM;
        }
        n->bytes += e.bytes;
    }
    n->err = umma_error_word();
    if (!n->err || cudaMallocHost(&n->host, sizeof(FarnetResult) + P * sizeof(float)) ||
        cudaFuncSetAttribute(k_t_lateral<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LAT_SMEM) ||
        cudaFuncSetAttribute(k_t_lateral<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LAT_SMEM) ||
        cudaFuncSetAttribute(k_t_operands, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OPERANDS_SMEM)) {
        mms_farnet_destroy(n);
        mms_set_error("mms_farnet_create: kernel set-up failed");
        return MMS_ERR_CUDA;
    }
    cudaMemset(n->w, 0, P * sizeof(float));
    k_t_fill<<<nblk(P), TB>>>(n->sc, P, 1.f);
    cudaMemset(n->m, 0, P * sizeof(float));
    cudaMemset(n->v, 0, P * sizeof(float));
    if (cudaMemcpy(n->lev_dev, n->lev_off, sizeof(n->lev_off), cudaMemcpyHostToDevice) != cudaSuccess) {
        mms_farnet_destroy(n);
        mms_set_error("mms_farnet_create: copy failed");
        return MMS_ERR_CUDA;
    }
    *out = n;
    return MMS_OK;
}

void mms_farnet_destroy(mms_farnet *n)
{
    if (!n) return;
    cudaDeviceSynchronize();
    void *b[] = {n->w, n->wt, n->sc, n->g, n->m, n->v, n->M, n->Lf, n->dM, n->dL, n->dout, n->lsum, n->res, n->ops, n->Cp,
                 n->lev_dev};
    for (void *p : b)
        if (p) cudaFree(p);
    if (n->host) cudaFreeHost(n->host);
    delete n;
}

int mms_farnet_set_weights(mms_farnet *n, const float *w, long long count)
{
    if (!n || !w || count != fn_num_params()) {
        mms_set_error("mms_farnet_set_weights: need %lld weights", fn_num_params());
        return MMS_ERR_ARG;
    }
    MMS_CUDA_TRY(cudaMemcpy(n->w, w, count * sizeof(float), cudaMemcpyHostToDevice));
    MMS_CUDA_TRY(cudaMemset(n->m, 0, count * sizeof(float)));
    MMS_CUDA_TRY(cudaMemset(n->v, 0, count * sizeof(float)));
    n->step = 0;
    return MMS_OK;
}

int mms_farnet_set_step_scale(mms_farnet *n, const float *scale, long long count)
{
    if (!n || !scale || count != fn_num_params()) {
        mms_set_error("mms_farnet_set_step_scale: need %lld scales", fn_num_params());
        return MMS_ERR_ARG;
    }
    MMS_CUDA_TRY(cudaMemcpy(n->sc, scale, count * sizeof(float), cudaMemcpyHostToDevice));
    return MMS_OK;
}

int mms_farnet_get_weights(mms_farnet *n, float *w, long long count)
{
    if (!n || !w || count != fn_num_params()) {
        mms_set_error("mms_farnet_get_weights: need %lld weights", fn_num_params());
        return MMS_ERR_ARG;
    }
    MMS_CUDA_TRY(cudaMemcpy(w, n->w, count * sizeof(float), cudaMemcpyDeviceToHost));
    return MMS_OK;
}

int mms_farnet_forward_dev(mms_farnet *n, const float *u, float *out, int nbatch)
{
    MMS_TRY(check_batch(n, nbatch));
    if (!u || !out) {
        mms_set_error("mms_farnet_forward_dev: NULL argument");
        return MMS_ERR_ARG;
    }
    MMS_TRY(forward(n, u, nbatch));
    k_t_leaf<false><<<div_up((long long)nbatch * n->nb * n->nb, LEAF_BOXES), FN_C>>>(
        n->w, n->Lf, out, nullptr, nullptr, nullptr, nullptr, netk(n, nbatch), nbatch);
    MMS_CUDA_TRY(cudaGetLastError());
    MMS_CUDA_TRY(cudaStreamSynchronize(0));
    return MMS_OK;
}

int mms_farnet_gradient(mms_farnet *n, const float *u, const float *far, const float *nrm2, int nbatch, float *grad,
                        double *loss)
{
    MMS_TRY(check_batch(n, nbatch));
    if (!u || !far || !nrm2) {
        mms_set_error("mms_farnet_gradient: NULL argument");
        return MMS_ERR_ARG;
    }
    return gradient(n, u, far, nrm2, nbatch, loss, grad);
}

int mms_farnet_train_step(mms_farnet *n, const float *u, const float *far, const float *nrm2, int nbatch, float lr,
                          float beta1, float beta2, float eps, double *loss)
{
    MMS_TRY(check_batch(n, nbatch));
    if (!u || !far || !nrm2 || !(lr >= 0)) {
        mms_set_error("mms_farnet_train_step: bad argument");
        return MMS_ERR_ARG;
    }
    MMS_TRY(gradient(n, u, far, nrm2, nbatch, loss, nullptr));
    n->step++;
    const float c1 = 1.f - powf(beta1, (float)n->step), c2 = 1.f - powf(beta2, (float)n->step);
    const long long P = fn_num_params();
    k_t_adam<<<nblk(P), TB>>>(n->w, n->g, n->m, n->v, n->sc, P, lr, beta1, beta2, eps, c1, c2);
    MMS_CUDA_TRY(cudaGetLastError());
    return MMS_OK;
}

long long mms_farnet_device_bytes(const mms_farnet *n) { return n ? (long long)n->bytes : 0; }

}  // extern "C"
