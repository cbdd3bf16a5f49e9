// The separable preconditioner of the pressure and velocity systems and the Krylov solves
// that use it.
//
// On the tensor-product pressure grid the operator of NavierStokes/kernels/LHS2.cu
// (dt D G) is A0 = X (x) I + I (x) Y with tridiagonal X (entries of the column spacing)
// and Y (of the row spacing), plus one or two doubled diagonals (the pinned cells) and,
// for the immersed-boundary methods that patch it, the rows at the body.  A0 is inverted
// directly: X = V diag(lambda) V^-1 with V = D^-1/2 Q, Q orthonormal (X is symmetric in
// the column widths D), so
//     r^ = Q^T D^1/2 r   (one dense product per row of the grid),
//     (Y + lambda_k) z^_k = r^_k   (one tridiagonal solve per mode k),
//     z = D^-1/2 Q z^    (the second dense product),
// and the pinned cells are a rank-two or rank-three correction (Woodbury) of z^ before
// the second product.  Q comes from the implicitly shifted QR iteration on the symmetric
// tridiagonal matrix (Golub and Van Loan, Matrix Computations, ch. 8.3): the rotations
// are found on the host in O(n^2) and applied to the identity on the GPU.
//
// Why: smoothed aggregation needed 70 to 330 BiCGSTAB iterations a step on the stretched,
// nearly singular operators of the cylinder grids (Re 550, 922 x 922, to 1e-13: 250
// iterations, 95 ms); this preconditioner is the inverse to rounding, so the solve ends
// after one application or two.  It stays a preconditioner of the same Krylov method, with
// the same stopping rule on the FP64 residual, so what the dense products' rounding leaves
// (about 1e-9 of the residual at 922 x 922, as FP64 products leave it) the iteration
// removes.  The velocity operator (I - dt/2 nu L, LHS1.cu) is 1 + X (x) I + I (x) Y on the u
// and on the v grid, without pinned cells; both grids go through the same launches.
//
// The dense products are 2 n_m^2 n_r multiply-adds each, which at GB300's FP64 rate
// (1.25 TFLOP/s) would take 1.25 ms at 922 x 922.  They run on the tensor cores instead,
// exactly: a row is scaled by a power of two and written as kDigits base-256 digits in
// [-128, 128] (55 bits below the row's largest value for 7 digits), each digit a BF16
// value, and the products of digit i of one factor with digit j of the other, i + j <
// kDigits, are accumulated as whole numbers below 2^24, which FP32 accumulators hold
// exactly; every 128 terms the sums of equal i + j go into one 64-bit integer.  What is
// dropped (i + j >= 7) is 2^-51 of the factors' row maxima: as little as the rounding of an FP64
// sum of terms of that size, but more than it where a row's terms are far below its maximum;
// the iteration on the FP64 residual takes out either (the splitting of Ozaki, Ogita, Oishi and
// Rump, Numer. Algorithms 59, 2012).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "krylov_device.cuh"
#include "separable.h"

namespace cuibm {

constexpr int kDigits = 7;       // digits of the FP64 solves: 28 products a dense product
// Mixed precision with a Fadlun body: 31 bits below the row's largest value, 10 products, and an
// application more.  The plain method's mixed solves take kDigits too: one application of 28
// products is cheaper than two of 10 (velocity, 64 x 64 71 against 131 us, 270 x 270 122 against
// 207, 512 x 512 217 against 307)
constexpr int kDigitsMixed = 4;
constexpr int kKC = 32;          // terms of a chunk of the dense product's sum
constexpr int kFlush = 4;        // chunks between flushes: 7 x 128 x 2^14 < 2^24
// Transforms up to this length; from there on the products (n_m^2 n_r) and the tables
// (28 n_m^2 bytes) outgrow what was measured, and the accumulators' range ends at 4096
constexpr int kSepMax = 2048;
constexpr int kTriThreads = 512;
constexpr int kRowPlaces = 400;  // the row kernels' longest rows (at most 512: two pairs a thread)

// Device view of one grid's plan.  The pressure system has one grid; the velocity system
// two (u, v), which every kernel takes in one launch.
struct SepDev {
    int nm, nr;            // modes (length of the transformed direction), rows (the other)
    int sm, sr, base;      // a field's layout: element (row R, place m) at base + R sr + m sm
    int nch;               // chunks of kKC terms in a transform
    const __nv_bfloat16 *B1, *B2;  // digits of Q^T and of Q
    const double *sB1, *sB2;       // their row scales (and the output's D^-1/2)
    __nv_bfloat16 *A;      // digits of the operand at hand
    double *sA;
    double *h;             // r^, then z^: [row][mode]
    const double *l, *c, *inv;     // tridiagonal factors [row][mode]
    const double *Pf, *Pb;         // products of l and c over a thread's rows [thread row][mode]
    const double *cm, *cr;         // input scaling per place and per row (cr null: 1)
    // the transposed inverse, W A0^-1 W^-1 with the cell areas W: its input scaling, the
    // transform back and its output scaling per row
    const double *cmt, *crt, *sB2t, *wr;
    // a moving body's rows (null: none): r is scaled there by the ratio of A0's diagonal to
    // the row's own
    RowPatch patch;
    const double *E, *W, *N, *S;
    int nx;
    // pinned cells (the pressure system): functionals F (rows R0, R1), responses G, the
    // constant's response gm
    int pins, R[2], k0;
    const double *F[2], *G[2], *gm;
    double K[9], mean;
};
// What tells the products of a solve's first application of the preconditioner that the vector
// the solve starts from meets the tolerance already (a steady flow): they end at once, and the
// kernels between them work on values that nothing looks at.  The flat kernels' start leaves the
// status.  The row kernels' start leaves its sums partial, and beside them their totals by
// atomic adds, in no fixed order.  Those are compared to 20 bits with room for that order and
// the bits left out, so that a closed gate is certain of the ordered sums too, which alone
// decide what the solve does (in FP32: FP64 products and a comparison in every warp cost more
// than the load).  A steady flow stops changing just below the tolerance - the last solve was
// the last residual above it - so a rough comparison would not see it.  A steady cavity's step
// at 128 x 128 takes 85 us with the gate and 103 without, an unsteady one's 1 us more than
// without; a gate in the other kernels too gave 72 and 2 to 7 us.  Null pointers: open.
struct SepGate {
    const int *status = nullptr;
    const double *acc = nullptr;  // ||r||^2, ||b||^2
    float m = 0;                  // rtol^2 = m 2^e, 1 <= m < 2
    int e = 0;
    // the leading 20 bits of a positive double, from its high word
    static __device__ __forceinline__ float mantissa(int high)
    {
        return __int_as_float((high & 0xfffff) << 3 | 0x3f800000);
    }
    // what a kernel loads at its start, and looks at after its own first loads are under way
    struct Seen {
        int r, b;
    };
    __device__ __forceinline__ Seen look() const
    {
        if (!acc) return Seen{status ? *status : KS_RUNNING, 0};
        const int *h = reinterpret_cast<const int *>(acc);  // (the high word is the second)
        return Seen{h[1], h[3]};
    }
    __device__ __forceinline__ bool closed(const Seen &s) const
    {
        if (!acc) return s.r != KS_RUNNING;
        const int d = min(max((s.b >> 20) + e - (s.r >> 20), -4), 4);
        return (s.b >> 20) > 0 & mantissa(s.r) <= m * mantissa(s.b) * __int_as_float((d + 127) << 23) * (1 - 1e-5f);
    }
};
// A solve's last correction (k_sep_accept) is left out where it failed or made no step.
__device__ __forceinline__ bool no_correction(const KrylovScalars *ks)
{
    return ks->status != KS_CONVERGED || !(ks->s_done || ks->body_runs);
}
struct SepArgs {
    SepDev f[2];
    SepGate gate;
};

struct SepPlan {
    SepArgs a{};
    int grids = 1;
    int digits = kDigits;
    char *block[2] = {nullptr, nullptr};  // one device allocation a grid
    // rows that a body patches (a fixed body's): how many, their cells, each cell's place in
    // that list (or -1), the inverse of the capacitance matrix, and work arrays
    int patched = 0;
    int *prow = nullptr, *pidx = nullptr;
    double *cap = nullptr, *gap = nullptr, *q = nullptr, *y = nullptr, *rin = nullptr;
    char *pblock = nullptr;
    // sums of the row kernels (k_row_*): six arrays of sums_cap, then SepGate::acc
    double *sums = nullptr;
    int sums_cap = 0;
    bool rows = false;    // their layout applies
    bool moving = false;  // a body's rows change: one Jacobi sweep on them beside A0^-1
    int tri_rows = 0;  // neighbouring rows a thread of k_sep_tri takes
    int max_nm() const { return grids > 1 ? std::max(a.f[0].nm, a.f[1].nm) : a.f[0].nm; }
    int max_nr() const { return grids > 1 ? std::max(a.f[0].nr, a.f[1].nr) : a.f[0].nr; }
    int first_kernels = 0;  // kernels of the conditional body after the first half iteration
};

// ---- the operators with their stored diagonal --------------------------------------------
// five FP64 operations a row instead of nine (the Krylov kernels are FP64-issue bound)
struct StoredOp2 {
    Lhs2Coef c;
    const double *diag, *w;
    int nx, ny;
    template <class X>
    __device__ __forceinline__ double row(int i, const X &x) const
    {
        double y;
        const int k = c.patch.pid ? c.patch.pid[i] : -1;
        if (k >= 0) {
            y = patch_row(c.patch, k, x(i), x);
        } else {
            const int J = i / nx, I = i - J * nx;
            y = diag[i] * x(i);
            if (I != nx - 1) y -= c.E[I] * x(i + 1);
            if (I != 0) y -= c.W[I] * x(i - 1);
            if (J != ny - 1) y -= c.N[J] * x(i + nx);
            if (J != 0) y -= c.S[J] * x(i - nx);
        }
        return w ? w[i] * y : y;
    }
};
struct StoredOp1 {  // without row scales (the methods other than the embedded one)
    Lhs1Coef c;
    const double *diag, *w;
    int nx, ny, nU;
    template <class X>
    __device__ __forceinline__ double row(int i, const X &x) const
    {
        const int pk = c.patch.pid ? c.patch.pid[i] : -1;
        if (pk >= 0) {
            const double yp = patch_row(c.patch, pk, x(i), x);
            return w ? w[i] * yp : yp;
        }
        const bool u = i < nU;
        const int n = u ? nx - 1 : nx, m = u ? ny : ny - 1, k = u ? i : i - nU, J = k / n, I = k - J * n;
        const double *E = u ? c.uE : c.vE, *W = u ? c.uW : c.vW, *N = u ? c.uN : c.vN, *S = u ? c.uS : c.vS;
        double y = diag[i] * x(i);
        if (I != n - 1) y -= E[I] * x(i + 1);
        if (I != 0) y -= W[I] * x(i - 1);
        if (J != m - 1) y -= N[J] * x(i + n);
        if (J != 0) y -= S[J] * x(i - n);
        return w ? w[i] * y : y;
    }
};

// ---- digits -------------------------------------------------------------------------
// base-256 digits, most significant first, of v scaled so that |v| < 2^(8 L - 1)
template <int L>
__device__ __forceinline__ void digits_of(double v, double scale, float (&dg)[L])
{
    long long x = __double2ll_rn(v * scale);
#pragma unroll
    for (int i = L - 1; i > 0; --i) {
        const int lo = (int)(signed char)(unsigned char)(x & 255);
        dg[i] = (float)lo;
        x = (x - lo) >> 8;
    }
    dg[0] = (float)(int)x;
}

// 2^k as a double, -1022 <= k <= 1023
__device__ __forceinline__ double pow2(int k) { return __longlong_as_double((long long)(k + 1023) << 52); }

// the power of two above a row's largest magnitude (its bits); false: not finite
__device__ __forceinline__ bool row_exponent(long long maxbits, int &e)
{
    const int be = (int)(maxbits >> 52);
    e = max(be, 122) - 1022;  // rows below 2^-900 count as zero
    return be < 0x7ff;
}

__device__ __forceinline__ long long block_max(long long v)
{
    __shared__ long long sh[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) sh[w] = v;
    __syncthreads();
    v = sh[lane < nw ? lane : 0];
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// A row of n values to digits: [chunk][digit][kKC], zero from n on to the end of the last
// chunk.  A thread holds pairs of neighbours, NP of them (places 2 (thread + q blockDim) and
// the next; zero from n on).  Returns the row's scale.
template <int L, int NP>
__device__ __forceinline__ double split_values(int n, int nch, __nv_bfloat16 *out, const double (&v)[2 * NP])
{
    long long mx = 0;
#pragma unroll
    for (int q = 0; q < 2 * NP; ++q) mx = max(mx, __double_as_longlong(fabs(v[q])));
    mx = block_max(mx);
    int e;
    const bool finite = row_exponent(mx, e);
    const double scale = finite ? pow2(8 * L - 1 - e) : 0.0;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const int m = 2 * (threadIdx.x + q * blockDim.x);
        if (m >= nch * kKC) break;
        float a[L], b[L];
        digits_of<L>(finite ? v[2 * q] : 0.0, scale, a);
        digits_of<L>(finite ? v[2 * q + 1] : 0.0, scale, b);
        __nv_bfloat16 *o = out + (size_t)(m / kKC) * (L * kKC) + m % kKC;
#pragma unroll
        for (int i = 0; i < L; ++i)
            *reinterpret_cast<__nv_bfloat162 *>(o + i * kKC) = __floats2bfloat162_rn(a[i], b[i]);
    }
    return finite ? pow2(e) : __longlong_as_double(0x7ff8000000000000ll);
}

template <int L, int NP, class Value>
__device__ __forceinline__ double split_row(int n, int nch, __nv_bfloat16 *out, const Value &value)
{
    double v[2 * NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        const int m = 2 * (threadIdx.x + q * blockDim.x);
        v[2 * q] = m < n ? value(m) : 0.0;
        v[2 * q + 1] = m + 1 < n ? value(m + 1) : 0.0;
    }
    return split_values<L, NP>(n, nch, out, v);
}

// rows of a table: src[r ld_r + m ld_m], the scale of row r times 2^-50 and extra[r]
template <int L, int NP>
__global__ void k_sep_split_table(const double *__restrict__ src, int n, int nch, int ld_r, int ld_m,
                                  const double *__restrict__ extra, __nv_bfloat16 *out, double *scale)
{
    const int r = blockIdx.x;
    const double s = split_row<L, NP>(n, nch, out + (size_t)r * nch * L * kKC,
                                      [&](int m) { return src[(size_t)r * ld_r + (size_t)m * ld_m]; });
    if (threadIdx.x == 0) scale[r] = s * pow2(-50) * (extra ? extra[r] : 1.0);
}

// A block's sums, the one of v[k] in every lane of warp k.  An FP64 warp instruction takes its
// quarter of an SM 64 cycles (two lanes a clock an SM; a square root 650, a division 570:
// measured), so that five shuffled adds a value in every warp cost more than the B / 32 + 5
// adds of one warp a value over shared memory.
template <int NV, int B>
__device__ __forceinline__ double block_total(const double (&v)[NV])
{
    static_assert(NV <= B / 32, "a warp a value");
    __shared__ double sh[NV][B];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();  // (sh may be in use by an earlier call)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][threadIdx.x] = v[k];
    __syncthreads();
    double a = 0;
    if (w < NV) {
#pragma unroll
        for (int j = 0; j < B / 32; ++j) a += sh[w][lane + 32 * j];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    }
    return a;
}

// the ratio of A0's diagonal to a patched row's own (1 for a row without one)
__device__ __forceinline__ double row_ratio(const SepDev &d, int i, int k)
{
    const double own = d.patch.pdiag[k];
    if (own == 0) return 1.0;
    const int J = i / d.nx, I = i - J * d.nx;
    return ((d.E[I] + d.W[I]) + (d.N[J] + d.S[J])) / own;
}

// One grid row to digits, a block a row.  SPEC false: a field (times the scaling that
// makes the transform orthonormal); true: z^, with the pinned cells' correction.  A row of
// 922 is 7 values a thread: bound by one round of loads, the conversion and the stores.
template <int L, int NP, bool SPEC>
__global__ void __launch_bounds__(128) k_sep_split(const __grid_constant__ SepArgs args, const double *__restrict__ in,
                                                   int transposed)
{
    const SepDev &d = args.f[blockIdx.y];
    const int R = blockIdx.x, n = d.nm;
    if (R >= d.nr) return;
    __nv_bfloat16 *out = d.A + (size_t)R * d.nch * L * kKC;
    double s;
    if (!SPEC) {
        const double *row = in + d.base + (size_t)R * d.sr;
        const double *cm = transposed ? d.cmt : d.cm, *crp = transposed ? d.crt : d.cr;
        const double cr = crp ? crp[R] : 1.0;
        if (d.patch.pid && !transposed)
            s = split_row<L, NP>(n, d.nch, out, [&](int m) {
                const int i = d.base + R * d.sr + m * d.sm, k = d.patch.pid[i];
                const double v = in[i] * (cm[m] * cr);
                return k >= 0 ? v * row_ratio(d, i, k) : v;
            });
        else
            s = split_row<L, NP>(n, d.nch, out, [&](int m) { return row[(size_t)m * d.sm] * (cm[m] * cr); });
    } else {
        const double *row = d.h + (size_t)R * n;
        if (d.pins == 0) {
            s = split_row<L, NP>(n, d.nch, out, [&](int m) { return row[m]; });
            if (threadIdx.x == 0) d.sA[R] = s;
            return;
        }
        // q = K^-1 (values of z at the pinned cells, mean of row 0), the same in every block;
        // both sums in one pass, with the row's own loads in flight
        const bool two = d.pins > 1;
        const double *g0 = d.G[0] + (size_t)R * n, *g1 = two ? d.G[1] + (size_t)R * n : g0;
        double own[2 * NP], r0[2 * NP], r1[2 * NP], f0 = 0, f1 = 0;
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u) {
            const int m = 2 * (threadIdx.x + (u >> 1) * blockDim.x) + (u & 1);
            own[u] = m < n ? row[m] : 0.0;
            r0[u] = m < n ? g0[m] : 0.0;
            r1[u] = m < n && two ? g1[m] : 0.0;
        }
        const double *h0 = d.h + (size_t)d.R[0] * n, *h1 = d.h + (size_t)d.R[two] * n;
        const double *F0 = d.F[0], *F1 = d.F[two];
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            f0 += F0[k] * h0[k];
            f1 += F1[k] * h1[k];
        }
        const double fm = d.h[d.k0] * d.mean, gm = d.gm[R], part[2] = {f0, f1};
        __shared__ double tot[2];
        const double total = block_total<2, 128>(part);
        if (threadIdx.x < 64 && threadIdx.x % 32 == 0) tot[threadIdx.x / 32] = total;
        __syncthreads();
        f0 = tot[0];
        f1 = tot[1];
        // f = (f0, f1, fm), without f1 for one pinned cell
        const double a1 = two ? f1 : fm, a2 = two ? fm : 0.0;
        const double q0 = d.K[0] * f0 + d.K[1] * a1 + d.K[2] * a2, q1 = d.K[3] * f0 + d.K[4] * a1 + d.K[5] * a2,
                     q2 = d.K[6] * f0 + d.K[7] * a1 + d.K[8] * a2;
        const double qm = (two ? q2 : q1) * gm, qg = two ? q1 : 0.0;
#pragma unroll
        for (int u = 0; u < 2 * NP; ++u) {
            const int m = 2 * (threadIdx.x + (u >> 1) * blockDim.x) + (u & 1);
            own[u] -= q0 * r0[u] + qg * r1[u];
            if (m == d.k0) own[u] += qm;
        }
        s = split_values<L, NP>(n, d.nch, out, own);
    }
    if (threadIdx.x == 0) d.sA[R] = s;
}

// ---- the dense product ------------------------------------------------------------------
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp16(unsigned dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}

// out(M, N) = A(M, K) B(N, K)^T from digits, WM x WN warps of 16 x 16 outputs.  A stage in
// shared memory is one chunk of the tile's rows of both factors, kKC terms of every digit;
// a row is 64 L + 16 bytes there, an odd number of 16-byte units, so ldmatrix meets no
// bank conflict.  A warp holds its L digit fragments of A and walks the digits of B: 2 L
// ldmatrix for L (L + 1) mma.  The bound is the latency between dependent instructions of few
// warps: with the next fragments and the copies to a later stage issued among the mma (and the
// copies' addresses formed once), a step of the mixed cavity 512 x 512 went from 556 to 517 us,
// Re 40 (270 x 270) from 377 to 364, a Poisson solve at 662 x 326 from 316 to 298.
template <int L, int WM, int WN, int ST>
__global__ void __launch_bounds__(32 * WM * WN, 2) k_sep_gemm(const __grid_constant__ SepArgs args,
                                                             double *__restrict__ field, int back)
{
    // back 0: h = (digits of the field) Q; 1: field = (digits of z^) Q^T; 2: the transposed inverse's
    const SepDev &d = args.f[blockIdx.z];
    const __nv_bfloat16 *__restrict__ A = d.A, *__restrict__ B = back ? d.B2 : d.B1;
    const double *__restrict__ sA = d.sA, *__restrict__ sB = back == 2 ? d.sB2t : back ? d.sB2 : d.sB1;
    const int M = d.nr, N = d.nm, nch = d.nch, so_m = back ? d.sr : d.nm, so_n = back ? d.sm : 1;
    double *__restrict__ out = back ? field + d.base : d.h;
    constexpr int TM = 16 * WM, TN = 16 * WN, T = 32 * WM * WN;
    constexpr int RB = 64 * L + 16;                // bytes of a row in a stage
    constexpr int STAGE = (TM + TN) * RB;
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    if (m0 >= M || n0 >= N) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp / WN, wn = warp % WN;
    const size_t rowBytes = (size_t)nch * L * kKC * 2;

    const SepGate::Seen seen = args.gate.look();
    // a thread's 16-byte units of a chunk: the same places in every stage
    constexpr int U = 4 * L, UNITS = (TM + TN) * U, CNT = (UNITS + T - 1) / T;
    const char *src[CNT];
    unsigned dst[CNT];
#pragma unroll
    for (int i = 0; i < CNT; ++i) {
        const int u = min((int)threadIdx.x + i * T, UNITS - 1), row = u / U, k = u - row * U;
        src[i] = (row < TM ? reinterpret_cast<const char *>(A) + (size_t)min(m0 + row, M - 1) * rowBytes
                           : reinterpret_cast<const char *>(B) + (size_t)min(n0 + row - TM, N - 1) * rowBytes) +
                 k * 16;
        dst[i] = sbase + row * RB + k * 16;
    }
    auto load = [&](int ch, int i) {
        if (UNITS % T == 0 || (int)threadIdx.x + i * T < UNITS)
            cp16(dst[i] + (ch % ST) * STAGE, src[i] + (size_t)ch * (U * 16));
    };

    float acc[L][2][4];
    long long tot[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) tot[t][q] = 0;
#pragma unroll
    for (int d = 0; d < L; ++d)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[d][t][q] = 0.f;

    for (int s = 0; s < ST - 1; ++s) {
        if (s < nch)
#pragma unroll
            for (int i = 0; i < CNT; ++i) load(s, i);
        asm volatile("cp.async.commit_group;");
    }
    if (args.gate.closed(seen)) {
        asm volatile("cp.async.wait_all;");
        return;
    }
    const unsigned offA = (wm * 16 + (lane & 15)) * RB + (lane >> 4) * 16;
    const unsigned offB = (TM + wn * 16 + (lane & 7) + ((lane >> 4) << 3)) * RB + ((lane >> 3) & 1) * 16;
    for (int ch = 0; ch < nch; ++ch) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2));
        __syncthreads();
        const unsigned s = sbase + (ch % ST) * STAGE;
        unsigned a[L][4], b[2][4];
#pragma unroll
        for (int i = 0; i < L; ++i) ldsm4(a[i], s + offA + i * 64);
        ldsm4(b[0], s + offB);
        // 2 L steps: the mma of one digit of B, 16 terms.  The next step's fragment of B, the
        // next 16 terms' fragment of A that this step was the last to need, and the step's share
        // of the copies to a later stage are issued among them.
#pragma unroll
        for (int st = 0; st < 2 * L; ++st) {
            const int ks = st / L, j = st % L;
            if (st + 1 < 2 * L) ldsm4(b[(st + 1) & 1], s + offB + (st + 1) % L * 64 + (st + 1) / L * 32);
#pragma unroll
            for (int i = L - j - 1; i >= 0; --i) {
                mma_bf16(acc[i + j][0], a[i], b[st & 1][0], b[st & 1][1]);
                mma_bf16(acc[i + j][1], a[i], b[st & 1][2], b[st & 1][3]);
                if (ks == 0 && i == L - j - 1) ldsm4(a[i], s + offA + i * 64 + 32);
            }
            if (ch + ST - 1 < nch)
#pragma unroll
                for (int i = st * CNT / (2 * L); i < (st + 1) * CNT / (2 * L); ++i) load(ch + ST - 1, i);
        }
        asm volatile("cp.async.commit_group;");
        if ((ch % kFlush) == kFlush - 1 || ch == nch - 1) {
            // whole numbers below 2^24: into units of 2^-36 of the leading digits' product
#pragma unroll
            for (int d = 0; d < L; ++d)
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int w = __float2int_rn(acc[d][t][q]);
                        acc[d][t][q] = 0.f;
                        const int sh = 36 - 8 * d;
                        if (sh >= 0) tot[t][q] += (long long)w * (1ll << (sh >= 0 ? sh : 0));
                        else tot[t][q] += (w + (1 << (-sh - 1 > 0 ? -sh - 1 : 0))) >> (sh < 0 ? -sh : 0);
                    }
        }
    }
    const int r0 = m0 + wm * 16 + (lane >> 2), c0 = n0 + wn * 16 + (lane & 3) * 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = r0 + (q >> 1) * 8;
        if (r >= M) continue;
        const double sa = back == 2 ? sA[r] * d.wr[r] : sA[r];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int col = c0 + t * 8 + (q & 1);
            if (col < N) out[(size_t)r * so_m + (size_t)col * so_n] = (double)tot[t][q] * (sa * sB[col]);
        }
    }
}

// ---- the tridiagonal solves -----------------------------------------------------------------
// A block of T threads solves CB modes; T / CB threads share a mode's rows, m = ceil(nr / that)
// neighbouring rows each.  Forward d_J = r_J + l_J d_J-1 and backward x_J = inv_J d_J + c_J
// x_J+1 are linear recurrences: each thread runs its rows from zero, the threads' ends are
// joined by a scan of affine maps in shared memory (the factors' products over a thread's
// rows are tables), and each thread runs its rows again from the true start.  922 rows in
// sequence would be 1844 dependent FP64 operations; this way it is 5 x 15 and two scans of
// 6 steps.  The bound is FP64 issue, 64 cycles a warp instruction on a quarter of an SM, and
// a scan's 4 instructions a step are work that the rows alone would not need: so as few
// threads a mode as the rows a thread can hold (16) allow.
template <int CB, int T>
__device__ __forceinline__ double tri_scan(double end, double prod, bool up, double *se, double *sp)
{
    // inclusive scan over q of x -> end + prod x, from q = 0 up or from the last down;
    // returns the value that enters this thread's rows
    constexpr int NQ = T / CB;
    const int tid = threadIdx.x, q = up ? tid / CB : NQ - 1 - tid / CB, step = up ? CB : -CB;
    int cur = 0;
    se[tid] = end;
    sp[tid] = prod;
    __syncthreads();
#pragma unroll
    for (int o = 1; o < NQ; o <<= 1) {
        const double *e = se + cur * T, *p = sp + cur * T;
        double *en = se + (cur ^ 1) * T, *pn = sp + (cur ^ 1) * T;
        double ee = e[tid], pp = p[tid];
        if (q >= o) {
            const int from = tid - o * step;
            ee += pp * e[from];
            pp *= p[from];
        }
        en[tid] = ee;
        pn[tid] = pp;
        cur ^= 1;
        __syncthreads();
    }
    const double in = q > 0 ? se[cur * T + tid - step] : 0.0;
    __syncthreads();
    return in;
}

// M: rows a thread holds in registers, every load of the kernel issued at its start (0: any
// number, the rows in shared memory and the tables read as they are needed).  512 x 512: 15
// us with the tables read in four rounds.
template <int CB, int M, int T>
__global__ void __launch_bounds__(T) k_sep_tri(const __grid_constant__ SepArgs args, int m)
{
    const SepDev &d = args.f[blockIdx.y];
    extern __shared__ double row[];  // M = 0: [m][thread]: r, then inv d
    __shared__ double se[2 * T], sp[2 * T];
    const int tid = threadIdx.x, n = d.nm;
    const int k = blockIdx.x * CB + tid % CB, q = tid / CB;
    const int J0 = min(q * m, d.nr), J1 = min(J0 + m, d.nr), cnt = k < n ? J1 - J0 : 0;
    const size_t at = (size_t)J0 * n + k;
    const double pf = k < n ? d.Pf[(size_t)q * n + k] : 0.0, pb = k < n ? d.Pb[(size_t)q * n + k] : 0.0;
    double x = 0;
    if constexpr (M > 0) {
        double r[M], l[M], iv[M], cc[M];
#pragma unroll
        for (int t = 0; t < M; ++t) {
            const bool on = t < cnt;
            const size_t j = at + (size_t)t * n;
            r[t] = on ? d.h[j] : 0.0;
            l[t] = on ? d.l[j] : 0.0;
            iv[t] = on ? d.inv[j] : 0.0;
            cc[t] = on ? d.c[j] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < M; ++t)
            if (t < cnt) x = r[t] + l[t] * x;
        x = tri_scan<CB, T>(x, pf, true, se, sp);
#pragma unroll
        for (int t = 0; t < M; ++t) {
            x = r[t] + l[t] * x;
            r[t] = x * iv[t];
        }
        x = 0;
#pragma unroll
        for (int t = M - 1; t >= 0; --t)
            if (t < cnt) x = r[t] + cc[t] * x;
        x = tri_scan<CB, T>(x, pb, false, se, sp);
#pragma unroll
        for (int t = M - 1; t >= 0; --t)
            if (t < cnt) {
                x = r[t] + cc[t] * x;
                d.h[at + (size_t)t * n] = x;
            }
    } else {
#pragma unroll 4
        for (int t = 0; t < cnt; ++t) {
            const double r = d.h[at + (size_t)t * n];
            row[t * T + tid] = r;
            x = r + d.l[at + (size_t)t * n] * x;
        }
        x = tri_scan<CB, T>(x, pf, true, se, sp);
#pragma unroll 4
        for (int t = 0; t < cnt; ++t) {
            x = row[t * T + tid] + d.l[at + (size_t)t * n] * x;
            row[t * T + tid] = x * d.inv[at + (size_t)t * n];
        }
        x = 0;
#pragma unroll 4
        for (int t = cnt - 1; t >= 0; --t) x = row[t * T + tid] + d.c[at + (size_t)t * n] * x;
        x = tri_scan<CB, T>(x, pb, false, se, sp);
#pragma unroll 4
        for (int t = cnt - 1; t >= 0; --t) {
            x = row[t * T + tid] + d.c[at + (size_t)t * n] * x;
            d.h[at + (size_t)t * n] = x;
        }
    }
}

// Wide blocks of modes (whole 64-byte segments) where enough of them fill the GPU and their
// rows fit shared memory; kTriRows rows are what 4 modes a block can hold
constexpr int kTriRows = 6400;
static int tri_modes(int nm, int nr) { return nm >= 600 && nr <= kTriRows / 2 ? 8 : 4; }
// Threads of a block of 4 modes: the fewest whose 32 or 64 threads a mode hold its rows.  Against
// 128 threads a mode at every size, a step of the cavity 64 x 64 196 -> 183 us, Re 40 (270 x
// 270) 390 -> 377, Fadlun (162 x 162) 409 -> 383, mixed cavity 512 x 512 567 -> 556, Poisson
// 662 x 326 324 -> 316; longer rows stay in shared memory
static int tri_threads(int nm, int nr)
{
    if (tri_modes(nm, nr) == 8) return kTriThreads;
    return nr <= 32 * 16 ? 128 : nr <= 64 * 16 ? 256 : kTriThreads;
}

// the factors of Y + lambda_k, one thread a mode, and their products over each thread's
// rows of k_sep_tri; the constant's mode gets reg on its first diagonal
__global__ void k_sep_factor(int nm, int nr, int nq, int m, const double *__restrict__ up,
                             const double *__restrict__ dn, const double *__restrict__ lam, double shift, int k0,
                             double reg, double *l, double *c, double *inv, double *Pf, double *Pb)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nm) return;
    double prev = 0;
    for (int J = 0; J < nr; ++J) {
        double dg = shift + (up[J] + dn[J] + lam[k]);
        if (k == k0 && J == 0) dg += reg;
        const double lj = J ? dn[J] * prev : 0.0;
        if (J) dg -= lj * up[J - 1];
        prev = 1.0 / dg;
        const size_t at = (size_t)J * nm + k;
        l[at] = lj;
        inv[at] = prev;
        c[at] = J + 1 < nr ? up[J] * prev : 0.0;
    }
    for (int q = 0; q < nq; ++q) {
        double pf = 1, pb = 1;
        for (int J = q * m; J < min((q + 1) * m, nr); ++J) {
            pf *= l[(size_t)J * nm + k];
            pb *= c[(size_t)J * nm + k];
        }
        Pf[(size_t)q * nm + k] = pf;
        Pb[(size_t)q * nm + k] = pb;
    }
}

// Q from the QR iteration's rotations: every row of Q is a unit vector to which all
// rotations are applied in order.  A warp takes a row and applies 32 sweeps at once as a
// pipeline: lane l applies sweep l, two elements behind lane l - 1.  A rotation of elements
// k, k + 1 takes the carried element a and the next one x to the finished c a + s x and the
// carried c x - s a, so a lane is a shift register that hands its finished element to the
// next lane a step later, and where its sweep has no rotation it passes elements on (c = 1,
// s = 0).  922 x 922 in 7 ms; one thread a row, a rotation after another, took 120 ms.
struct Sweep {
    int first, count;
    long long at;
};
constexpr int kRotWarps = 8;
__global__ void __launch_bounds__(32 * kRotWarps) k_sep_rotate(int n, const Sweep *__restrict__ sw, int nsw,
                                                               const double2 *__restrict__ rot,
                                                               double *__restrict__ Q)
{
    extern __shared__ double rows[];
    const int lane = threadIdx.x & 31, i = blockIdx.x * kRotWarps + (threadIdx.x >> 5);
    if (i >= n) return;
    double *z = rows + (size_t)(threadIdx.x >> 5) * n;
    for (int j = lane; j < n; j += 32) z[j] = j == i ? 1.0 : 0.0;
    __syncwarp();
    for (int s0 = 0; s0 < nsw; s0 += 32) {
        const bool on = s0 + lane < nsw;
        const int lo = on ? sw[s0 + lane].first : 0, cnt = on ? sw[s0 + lane].count : 0;
        const double2 *r = rot + (on ? sw[s0 + lane].at : 0);
        double a = 0, out = 0;
        for (int t = 0; t < n + 63; ++t) {
            const int k = t - 2 * lane - 1 - lo;  // this step's rotation in the sweep
            double x = __shfl_up_sync(0xffffffffu, out, 1);
            if (lane == 0) x = t < n ? z[t] : 0.0;
            const double2 cs = k >= 0 && k < cnt ? r[k] : make_double2(1.0, 0.0);
            out = fma(cs.y, x, cs.x * a);
            a = fma(-cs.y, a, cs.x * x);
            if (lane == 31 && t >= 63) z[t - 63] = out;
        }
        __syncwarp();
    }
    for (int j = lane; j < n; j += 32) Q[(size_t)i * n + j] = z[j];
}

// column k0 of Q: the constant in exact form
__global__ void k_sep_constant(int n, int k0, const double *__restrict__ v, double *Q)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) Q[(size_t)i * n + k0] = v[i];
}

// ---- Krylov kernels ---------------------------------------------------------------------
// The rows of a grid of at most kRowBlocks blocks, and its sums: a block's partial sums go
// to memory, and the last block to arrive adds them in a fixed order with one warp.  The
// totals are valid in the last block's thread 0 (true there only).
static int row_blocks(int n) { return std::min(kRowBlocks, blocks_for(n)); }
#define SEP_ROWS(i, n) for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

// a block's sums to its places of the partial sums
// (acc: and added to NV totals, in the order the blocks come)
template <int NV, int B>
__device__ __forceinline__ void partial_store(const double (&v)[NV], double *p, int cap, int slot, double *acc = nullptr)
{
    const double a = block_total<NV, B>(v);
    const int w = threadIdx.x >> 5;
    if (w < NV && threadIdx.x % 32 == 0) {
        p[(size_t)w * cap + slot] = a;
        if (acc) atomicAdd(acc + w, a);
    }
}
// the same, and the last of the n blocks gets the totals (true in its thread 0)
template <int NV, int B>
__device__ __forceinline__ bool partial_last(double (&v)[NV], double *p, int cap, int slot, int n, unsigned int *arrive)
{
    __shared__ bool last;
    __shared__ double tot[NV];
    const int w = threadIdx.x >> 5;
    partial_store<NV, B>(v, p, cap, slot);
    if (w < NV && threadIdx.x % 32 == 0) __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(arrive, 1u) == (unsigned)n - 1;
        __threadfence();
    }
    __syncthreads();
    if (!last) return false;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        v[k] = 0;
        for (int b = threadIdx.x; b < n; b += B) v[k] += __ldcg(p + (size_t)k * cap + b);
    }
    const double a = block_total<NV, B>(v);
    if (w < NV && threadIdx.x % 32 == 0) tot[w] = a;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = tot[k];
    if (threadIdx.x == 0) *arrive = 0;
    return threadIdx.x == 0;
}
template <int NV>
__device__ __forceinline__ bool row_sums(double (&v)[NV], double *partials, unsigned int *arrive)
{
    return partial_last<NV, kBlock>(v, partials, kRowBlocks, blockIdx.x, gridDim.x, arrive);
}

// BiCGSTAB as in krylov.cu with two differences: the first half iteration takes r for its
// shadow residual and direction (they are copies then), and x takes alpha M p in the half
// step, so that a solve that ends there - the usual end - needs nothing more.
template <class Op>
__global__ void __launch_bounds__(256) k_sep_init(Op A, int n, const double *__restrict__ b, const double *x, double *r,
                                                  double *partials, KrylovScalars *ks, int *err, int which)
{
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double bi = b[i], ri = bi - A.row(i, PtrAccess{x});
        r[i] = ri;
        v[0] += ri * ri;
        v[1] += bi * bi;
    }
    if (row_sums<2>(v, partials, &ks->arrive)) {
        ks->rho = v[0];
        ks->rnorm = sqrt(v[0]);
        ks->bnorm = sqrt(v[1]);
        ks->tol = ks->rtol * ks->bnorm;
        ks->it = 0;
        ks->s_done = 0;
        ks->body_runs = 0;
        ks->status = KS_RUNNING;
        finish_status(ks, err, which);
    }
}

template <class Op>
__global__ void __launch_bounds__(256) k_sep_1(Op A, int n, const double *__restrict__ Mp, double *AMp,
                                               const double *__restrict__ rs, double *partials, KrylovScalars *ks,
                                               int first)
{
    if (ks->status != KS_RUNNING) return;
    double v[1] = {0};
    SEP_ROWS(i, n)
    {
        const double a = A.row(i, PtrAccess{Mp});
        AMp[i] = a;
        v[0] += rs[i] * a;
    }
    if (row_sums<1>(v, partials, &ks->arrive)) {
        ks->alpha = ks->rho / v[0];
        ks->s_done = 0;
        if (!first) ks->body_runs += 1;
    }
}

__global__ void __launch_bounds__(256) k_sep_2(int n, const double *__restrict__ r, const double *__restrict__ AMp,
                                               const double *__restrict__ Mp, double *s, double *x, double *partials,
                                               KrylovScalars *ks, int first, cudaGraphConditionalHandle h, int use_cond)
{
    if (ks->status != KS_RUNNING) return;
    const double alpha = ks->alpha;
    double v[1] = {0};
    SEP_ROWS(i, n)
    {
        const double si = r[i] - alpha * AMp[i];
        s[i] = si;
        x[i] += alpha * Mp[i];
        v[0] += si * si;
    }
    if (row_sums<1>(v, partials, &ks->arrive)) {
        ks->snorm = sqrt(v[0]);
        if (ks->snorm <= ks->tol) {
            ks->s_done = 1;
            ks->rnorm = ks->snorm;
            ks->status = KS_CONVERGED;
        } else if (first) {
            ks->body_runs = 1;
        }
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

template <class Op>
__global__ void __launch_bounds__(256) k_sep_3(Op A, int n, const double *__restrict__ s,
                                               const double *__restrict__ Ms, double *AMs, double *partials,
                                               KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double a = A.row(i, PtrAccess{Ms});
        AMs[i] = a;
        v[0] += a * s[i];
        v[1] += a * a;
    }
    if (row_sums<2>(v, partials, &ks->arrive)) ks->omega = v[0] / v[1];
}

// x += omega M s, r = s - omega A M s; the first time also rs = p = the residual the solve began with
__global__ void __launch_bounds__(256) k_sep_4(int n, double *x, double *r, double *rs, double *p,
                                               const double *__restrict__ s, const double *__restrict__ Ms,
                                               const double *__restrict__ AMs, double *partials, KrylovScalars *ks,
                                               int *err, int which, int first, cudaGraphConditionalHandle h,
                                               int use_cond)
{
    if (ks->status != KS_RUNNING) return;
    const double omega = ks->omega;
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double r0 = first ? r[i] : rs[i];
        if (first) {
            rs[i] = r0;
            p[i] = r0;
        }
        x[i] += omega * Ms[i];
        const double ri = s[i] - omega * AMs[i];
        r[i] = ri;
        v[0] += r0 * ri;
        v[1] += ri * ri;
    }
    if (row_sums<2>(v, partials, &ks->arrive)) {
        ks->beta = (v[0] / ks->rho) * (ks->alpha / omega);
        ks->rho = v[0];
        ks->it += 1;
        ks->rnorm = sqrt(v[1]);
        finish_status(ks, err, which);
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

// ---- the first iteration by rows ------------------------------------------------------------
// Where the transform runs along a field's contiguous direction, the first iteration's vector
// kernels take a block a row, as the splitting into digits does, and hand the digits of the
// vector they form straight on.  Their sums and those of the operator kernels between them
// stay partial: the kernel that needs a total adds the partials itself, in every block and in
// the same order (about 1 us, in place of a fence, an atomic and a last block's sum at the
// end of the kernel before: 4 to 6 us of a 10 us kernel at 270 x 270).  Only the kernels that
// decide how the solve goes on end with a last block.
struct RowSums {
    double *sums;
    int cap, ns, nr;  // partials of the starting kernel, of the operator kernels
};
// the sum of n partials, by one warp, in every lane
__device__ __forceinline__ double partial_total(const double *p, int n)
{
    double a = 0;
#pragma unroll 4
    for (int i = threadIdx.x % 32; i < n; i += 32) a += p[i];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

#define ROW_PLACES(u, m) \
    _Pragma("unroll") for (int u = 0, m = 2 * threadIdx.x; u < 2 * NP; ++u, m = 2 * (threadIdx.x + (u >> 1) * 128) + (u & 1))

// r = b - A x (CG: of the system with the cell areas), its digits and ||r||^2, ||b||^2
template <class Op, int L, int NP, bool CG>
__global__ void __launch_bounds__(128) k_row_start(const __grid_constant__ SepArgs args, Op A,
                                                   const double *__restrict__ b, const double *x, double *r, RowSums S)
{
    const SepDev &d = args.f[blockIdx.y];
    const int R = blockIdx.x, n = d.nm;
    if (R >= d.nr) return;  // (its partials stay the zeros they are set to)
    const double cr = d.cr ? d.cr[R] : 1.0;
    double v[2 * NP], t[2] = {0, 0};
    ROW_PLACES(u, m)
    {
        v[u] = 0;
        if (m < n) {
            const int i = d.base + R * d.sr + m;
            const double bi = b[i], ri = (CG ? A.w[i] * bi : bi) - A.row(i, PtrAccess{x});
            const double ro = CG ? ri / A.w[i] : ri;
            r[i] = ri;
            t[0] += ro * ro;
            t[1] += bi * bi;
            v[u] = ri * (d.cm[m] * cr);
        }
    }
    partial_store<2, 128>(t, S.sums, S.cap, blockIdx.y * gridDim.x + R, S.sums + 6 * (size_t)S.cap);
    const double e = split_values<L, NP>(n, d.nch, d.A + (size_t)R * d.nch * L * kKC, v);
    if (threadIdx.x == 0) d.sA[R] = e;
}

// a = A z and the partial sums y . a (TWO: and a . a; CG: and z . a with p = z)
template <class Op, int KIND>
__global__ void __launch_bounds__(256) k_row_apply(Op A, int n, const double *__restrict__ z, double *a,
                                                   const double *__restrict__ y, double *p, RowSums S, int at)
{
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double ai = A.row(i, PtrAccess{z}), yi = y[i];
        a[i] = ai;
        if (KIND == 2) {
            const double zi = z[i];
            p[i] = zi;
            v[0] += yi * zi;
            v[1] += zi * ai;
        } else {
            v[0] += yi * ai;
            if (KIND == 1) v[1] += ai * ai;
        }
    }
    partial_store<2, kBlock>(v, S.sums + (size_t)at * S.cap, S.cap, blockIdx.x);
}

// the gate's totals back to zero for the next solve's start, by the kernel that decides on the
// solve's first application (nothing after it in the solve looks at them)
__device__ __forceinline__ void row_reset(const RowSums &S)
{
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) S.sums[6 * (size_t)S.cap + threadIdx.x] = 0;
}
// What a solve starts with, from the starting kernel's sums (false: it ends there), and its
// first alpha, from the NA sums of the operator kernel.  A warp a sum, then a warp a square
// root or division, once a block.
template <int NA>
__device__ __forceinline__ bool row_begin(const RowSums &S, const KrylovScalars *ks, KrylovScalars &k)
{
    __shared__ double tot[2 + NA], fin[3];
    const int w = threadIdx.x >> 5;
    const bool head = threadIdx.x % 32 == 0;
    k = *ks;
    if (w < 2 + NA) {
        const double a = partial_total(S.sums + (size_t)w * S.cap, w < 2 ? S.ns : S.nr);
        if (head) tot[w] = a;
    }
    __syncthreads();
    if (w == 0 && head) fin[0] = sqrt(tot[0]);
    if (w == 1 && head) fin[1] = sqrt(tot[1]);
    if (w == 2 && head) fin[2] = NA == 1 ? tot[0] / tot[2] : tot[2] / tot[1 + NA];
    __syncthreads();
    k.rho = tot[0];
    k.rnorm = fin[0];
    k.bnorm = fin[1];
    k.tol = k.rtol * k.bnorm;
    k.it = k.s_done = k.body_runs = 0;
    k.status = KS_RUNNING;
    if (!(isfinite(k.rnorm) && isfinite(k.tol) && k.rnorm > k.tol && k.maxit > 0)) return false;
    if (NA == 2) k.rho = tot[2];
    k.alpha = fin[2];
    return true;
}
__device__ __forceinline__ void row_keep(KrylovScalars *ks, const KrylovScalars &k)
{
    ks->rho = k.rho;
    ks->alpha = k.alpha;
    ks->rnorm = k.rnorm;
    ks->bnorm = k.bnorm;
    ks->tol = k.tol;
    ks->snorm = k.snorm;
    ks->it = k.it;
    ks->s_done = k.s_done;
    ks->body_runs = k.body_runs;
    ks->status = k.status;
}

// s = r - alpha A M p, x += alpha M p, the digits of s; the solve may end here
template <int L, int NP>
__global__ void __launch_bounds__(128) k_row_half(const __grid_constant__ SepArgs args, const double *__restrict__ r,
                                                  const double *__restrict__ AMp, const double *__restrict__ Mp,
                                                  double *s, double *x, RowSums S, KrylovScalars *ks, int *err,
                                                  int which, cudaGraphConditionalHandle h, int use_cond)
{
    const SepDev &d = args.f[blockIdx.y];
    const int R = blockIdx.x, n = R < d.nr ? d.nm : 0;
    row_reset(S);
    KrylovScalars k;
    // the row's loads are under way while the sums are formed
    double ri[2 * NP], ai[2 * NP], zi[2 * NP], xi[2 * NP], ci[2 * NP];
    ROW_PLACES(u, m)
    {
        const bool in = m < n;
        const int i = d.base + R * d.sr + m;
        ri[u] = in ? r[i] : 0.0;
        ai[u] = in ? AMp[i] : 0.0;
        zi[u] = in ? Mp[i] : 0.0;
        xi[u] = in ? x[i] : 0.0;
        ci[u] = in ? d.cm[m] : 0.0;
    }
    if (!row_begin<1>(S, ks, k)) {
        if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
            row_keep(ks, k);
            finish_status(ks, err, which);
            set_cond(h, use_cond, 0);
        }
        return;
    }
    const double cr = d.cr && n ? d.cr[R] : 1.0;
    double v[2 * NP], q[1] = {0};
    ROW_PLACES(u, m)
    {
        v[u] = 0;
        if (m < n) {
            const int i = d.base + R * d.sr + m;
            const double si = ri[u] - k.alpha * ai[u];
            s[i] = si;
            x[i] = xi[u] + k.alpha * zi[u];
            q[0] += si * si;
            v[u] = si * (ci[u] * cr);
        }
    }
    if (n) {
        const double e = split_values<L, NP>(n, d.nch, d.A + (size_t)R * d.nch * L * kKC, v);
        if (threadIdx.x == 0) d.sA[R] = e;
    }
    if (partial_last<1, 128>(q, S.sums + 4 * (size_t)S.cap, S.cap, blockIdx.y * gridDim.x + R, gridDim.x * gridDim.y,
                        &ks->arrive)) {
        k.snorm = sqrt(q[0]);
        if (k.snorm <= k.tol) {
            k.s_done = 1;
            k.rnorm = k.snorm;
            k.status = KS_CONVERGED;
        } else {
            k.body_runs = 1;
        }
        row_keep(ks, k);
        set_cond(h, use_cond, k.status == KS_RUNNING);
    }
}

// x += omega M s, r = s - omega A M s, rs = p = the residual the solve began with
__global__ void __launch_bounds__(256) k_row_end(int n, double *x, double *r, double *rs, double *p,
                                                 const double *__restrict__ s, const double *__restrict__ Ms,
                                                 const double *__restrict__ AMs, RowSums S, KrylovScalars *ks, int *err,
                                                 int which, cudaGraphConditionalHandle h, int use_cond)
{
    __shared__ double o[2], quotient;
    const int w = threadIdx.x >> 5;
    if (w < 2) {
        const double a = partial_total(S.sums + (size_t)(2 + w) * S.cap, S.nr);
        if (threadIdx.x % 32 == 0) o[w] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) quotient = o[0] / o[1];
    __syncthreads();
    const double omega = quotient;
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double r0 = r[i];
        rs[i] = r0;
        p[i] = r0;
        x[i] += omega * Ms[i];
        const double ri = s[i] - omega * AMs[i];
        r[i] = ri;
        v[0] += r0 * ri;
        v[1] += ri * ri;
    }
    if (partial_last<2, kBlock>(v, S.sums + 4 * (size_t)S.cap, S.cap, blockIdx.x, gridDim.x, &ks->arrive)) {
        ks->omega = omega;
        ks->beta = (v[0] / ks->rho) * (ks->alpha / omega);
        ks->rho = v[0];
        ks->it += 1;
        ks->rnorm = sqrt(v[1]);
        finish_status(ks, err, which);
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

// CG: x += alpha p, r -= alpha q, the digits of r; first: alpha from the sums before it
template <int L, int NP>
__global__ void __launch_bounds__(128) k_row_cg(const __grid_constant__ SepArgs args, const double *__restrict__ w,
                                                const double *__restrict__ p, const double *__restrict__ q, double *r,
                                                double *x, RowSums S, KrylovScalars *ks, int *err, int which, int first,
                                                cudaGraphConditionalHandle h, int use_cond)
{
    const SepDev &d = args.f[blockIdx.y];
    const int R = blockIdx.x, n = R < d.nr ? d.nm : 0;
    KrylovScalars k;
    if (first) {
        row_reset(S);
        if (!row_begin<2>(S, ks, k)) {
            if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
                row_keep(ks, k);
                finish_status(ks, err, which);
                set_cond(h, use_cond, 0);
            }
            return;
        }
    } else {
        k = *ks;
        if (k.status != KS_RUNNING) return;
    }
    const double cr = d.cr && n ? d.cr[R] : 1.0;
    double v[2 * NP], t[1] = {0};
    ROW_PLACES(u, m)
    {
        v[u] = 0;
        if (m < n) {
            const int i = d.base + R * d.sr + m;
            x[i] += k.alpha * p[i];
            const double ri = r[i] - k.alpha * q[i], ro = ri / w[i];
            r[i] = ri;
            t[0] += ro * ro;
            v[u] = ri * (d.cm[m] * cr);
        }
    }
    if (n) {
        const double e = split_values<L, NP>(n, d.nch, d.A + (size_t)R * d.nch * L * kKC, v);
        if (threadIdx.x == 0) d.sA[R] = e;
    }
    if (partial_last<1, 128>(t, S.sums + 4 * (size_t)S.cap, S.cap, blockIdx.y * gridDim.x + R, gridDim.x * gridDim.y,
                        &ks->arrive)) {
        k.it += 1;
        k.rnorm = sqrt(t[0]);
        row_keep(ks, k);
        finish_status(ks, err, which);
        set_cond(h, use_cond, ks->status == KS_RUNNING);
    }
}

// A last correction x += M r for the residual that the solve ends with (a moving body's
// solves): where the iteration stops, the level of the pressure - fixed by one pinned cell -
// carries up to 2e-9 of it at a relative residual of 1e-12; M resolves it exactly.  With the
// body's rows M is no more than near the inverse, and r - A M r can be the larger residual:
// the whole update is taken where that meets the solve's tolerance, else the length of it that
// leaves the least residual, which is never above the one that the solve ended with.
__global__ void k_sep_pick(int n, const double *__restrict__ r, const double *__restrict__ s, double *out,
                           KrylovScalars *ks)
{
    const bool skip = no_correction(ks);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) ks->skip = skip;
    if (!skip && i < n) out[i] = ks->s_done ? s[i] : r[i];
}
template <class Op>
__global__ void __launch_bounds__(256) k_sep_accept(Op A, int n, const double *__restrict__ r,
                                                    const double *__restrict__ z, double *partials, KrylovScalars *ks)
{
    if (ks->skip) return;
    double v[3] = {0, 0, 0};
    SEP_ROWS(i, n)
    {
        const double ri = r[i], ai = A.row(i, PtrAccess{z}), left = ri - ai;
        v[0] += left * left;
        v[1] += ri * ai;
        v[2] += ai * ai;
    }
    if (row_sums<3>(v, partials, &ks->arrive)) {
        const double left = sqrt(v[0]);
        if (left <= ks->tol) {
            ks->alpha = 1;
            ks->rnorm = left;
        } else {
            const double a = v[1] / v[2], rr = ks->rnorm * ks->rnorm;
            ks->alpha = isfinite(a) ? a : 0.0;
            ks->rnorm = sqrt(fmax(0.0, rr - ks->alpha * v[1]));
        }
    }
}
__global__ void k_sep_correct(int n, const double *__restrict__ z, double *x, const KrylovScalars *ks)
{
    if (ks->skip) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += ks->alpha * z[i];
}

// CG's first iteration: p = z, q = A z, rho = r . z, alpha = rho / (z . q)
template <class Op>
__global__ void __launch_bounds__(256) k_sep_cg_1(Op A, int n, const double *__restrict__ r,
                                                  const double *__restrict__ z, double *p, double *q,
                                                  double *partials, KrylovScalars *ks)
{
    if (ks->status != KS_RUNNING) return;
    double v[2] = {0, 0};
    SEP_ROWS(i, n)
    {
        const double zi = z[i], qi = A.row(i, PtrAccess{z});
        p[i] = zi;
        q[i] = qi;
        v[0] += r[i] * zi;
        v[1] += zi * qi;
    }
    if (row_sums<2>(v, partials, &ks->arrive)) {
        ks->rho = v[0];
        ks->alpha = v[0] / v[1];
    }
}

// ---- host side: set-up ------------------------------------------------------------------
namespace {

// Eigenvalues (d, on return) of the symmetric tridiagonal matrix with diagonal d and
// off-diagonal e, by implicitly shifted QR sweeps; the rotations of every sweep are
// recorded in order (element j and j + 1 of a row vector take c, s: [c a + s b, c b - s a]).
// False: no convergence (non-finite entries).
bool tridiagonal_qr(std::vector<double> &d, std::vector<double> e, std::vector<Sweep> &sweeps,
                    std::vector<double2> &rot)
{
    const int n = (int)d.size();
    const double eps = 2.220446049250313e-16;
    int hi = n - 1;
    for (long guard = 0; hi > 0; ++guard) {
        if (guard > 60L * n) return false;
        auto small = [&](int k) { return std::fabs(e[k]) <= eps * (std::fabs(d[k]) + std::fabs(d[k + 1])); };
        if (small(hi - 1)) {
            e[--hi] = 0;
            continue;
        }
        int lo = hi - 1;
        while (lo > 0 && !small(lo - 1)) --lo;
        // Wilkinson's shift: the eigenvalue of the trailing 2 x 2 block nearer its last entry
        const double g = 0.5 * (d[hi - 1] - d[hi]), b = e[hi - 1];
        const double mu = d[hi] - b * (b / (g + std::copysign(std::hypot(g, b), g)));
        if (!std::isfinite(mu)) return false;
        sweeps.push_back({lo, hi - lo, (long long)rot.size()});
        double x = d[lo] - mu, z = e[lo];
        for (int k = lo; k < hi; ++k) {
            const double r = std::sqrt(x * x + z * z);
            const double cc = r > 0 ? x / r : 1.0, ss = r > 0 ? z / r : 0.0;
            if (k > lo) e[k - 1] = r;
            const double a = d[k], w = d[k + 1], f = e[k];
            const double t = cc * ss * f * 2;
            d[k] = cc * cc * a + t + ss * ss * w;
            d[k + 1] = ss * ss * a - t + cc * cc * w;
            e[k] = cc * ss * (w - a) + (cc * cc - ss * ss) * f;
            if (k + 1 < hi) {
                x = e[k];
                z = ss * e[k + 1];
                e[k + 1] *= cc;
            }
            rot.push_back(make_double2(cc, ss));
        }
    }
    return true;
}

// the inverse of the leading n x n block (n <= 3) of K, rows of 3, by elimination with pivoting;
// false: singular or not finite
bool invert3(double *K, int n)
{
    double a[3][6] = {};
    for (int i = 0; i < n; ++i) {
        for (int j = 0; j < n; ++j) a[i][j] = K[3 * i + j];
        a[i][n + i] = 1;
    }
    for (int k = 0; k < n; ++k) {
        int p = k;
        for (int i = k + 1; i < n; ++i)
            if (std::fabs(a[i][k]) > std::fabs(a[p][k])) p = i;
        if (!(std::fabs(a[p][k]) > 0)) return false;
        for (int j = 0; j < 2 * n; ++j) std::swap(a[k][j], a[p][j]);
        const double s = 1 / a[k][k];
        for (int j = 0; j < 2 * n; ++j) a[k][j] *= s;
        for (int i = 0; i < n; ++i)
            if (i != k) {
                const double f = a[i][k];
                for (int j = 0; j < 2 * n; ++j) a[i][j] -= f * a[k][j];
            }
    }
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) {
            K[3 * i + j] = a[i][n + j];
            if (!std::isfinite(K[3 * i + j])) return false;
        }
    return true;
}

}  // namespace

// ---- the diagnostic trace -----------------------------------------------------------------
// With the option trace_solve a solve's launches are stamped as the persistent solves' barriers
// are: after each of them one thread writes the global timer and the line of the stamp in this
// file (top bit of the site set, to tell it from a line of fused_kernels.cuh).  A phase is then
// its kernels, the gaps between them and the stamp's own launch.
__global__ void k_sep_stamp(unsigned long long *trace, int site)
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    t &= 0xffffffffffffull;
    const unsigned long long k = site ? trace[0] + 1 : 1;  // (site 0: the solve's start)
    if (k >= (unsigned long long)kTraceLen) return;
    trace[k] = (unsigned long long)(site & 0xffff) << 48 | t;
    trace[0] = k;
}
static void stamp_site(Context &c, int site)
{
    if (!c.trace_which) return;
    k_sep_stamp<<<1, 1, 0, c.stream>>>(c.solve_trace + (c.trace_which - 1) * kTraceLen, site);
    CUIBM_TRY(cudaGetLastError());
}
static void stamp(Context &c, int line = __builtin_LINE()) { stamp_site(c, 0x8000 | line); }
// stamps for the solve launched while it lives
struct Traced {
    Context &c;
    Traced(Context &c_, int which) : c(c_)
    {
        c.trace_which = c.trace_solve ? which : 0;
        stamp_site(c, 0);
    }
    ~Traced() { c.trace_which = 0; }
};

template <int L, int WM, int WN, int ST>
static void launch_gemm_t(Context &c, const SepPlan &P, double *field, int back)
{
    constexpr int smem = ST * 16 * (WM + WN) * (64 * L + 16);
    const dim3 grid((P.max_nm() + 16 * WN - 1) / (16 * WN), (P.max_nr() + 16 * WM - 1) / (16 * WM), P.grids);
    k_sep_gemm<L, WM, WN, ST><<<grid, 32 * WM * WN, smem, c.stream>>>(P.a, field, back);
    CUIBM_TRY(cudaGetLastError());
}

template <class K>
static void allow_smem(K *fn, size_t bytes)
{
    CUIBM_TRY(cudaFuncSetAttribute(reinterpret_cast<const void *>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)bytes));
}

// once per context (set-up): dynamic shared memory above 48 KB.  The attribute is the process's,
// so every context sets the same value, the most that any case asks for: another thread's
// context, of another size, may set it between this one's call and launch.
template <int L>
static void allow_gemm()
{
    allow_smem(k_sep_gemm<L, 2, 2, 3>, 3 * 16 * 4 * (64 * L + 16));
    allow_smem(k_sep_gemm<L, 2, 4, 2>, 2 * 16 * 6 * (64 * L + 16));
}

// Tiles of 32 x 64 (two blocks an SM) where there are enough of them for every SM, else 32
// x 32: a 270 x 270 product is 81 small tiles or 45 large ones on 152 SMs
template <int L>
static void launch_gemm(Context &c, const SepPlan &P, double *field, int back)
{
    if (P.grids * ((P.max_nr() + 31) / 32) * ((P.max_nm() + 63) / 64) >= 152)
        launch_gemm_t<L, 2, 4, 2>(c, P, field, back);
    else
        launch_gemm_t<L, 2, 2, 3>(c, P, field, back);
}

template <int L, bool SPEC>
static void launch_split(Context &c, const SepPlan &P, const double *in, int tr = 0)
{
    const int n = (P.max_nm() + kKC - 1) / kKC * kKC;
    const dim3 grid(P.max_nr(), P.grids);
    if (n <= 256) k_sep_split<L, 1, SPEC><<<grid, 128, 0, c.stream>>>(P.a, in, tr);
    else if (n <= 512) k_sep_split<L, 2, SPEC><<<grid, 128, 0, c.stream>>>(P.a, in, tr);
    else if (n <= 1024) k_sep_split<L, 4, SPEC><<<grid, 128, 0, c.stream>>>(P.a, in, tr);
    else k_sep_split<L, 8, SPEC><<<grid, 128, 0, c.stream>>>(P.a, in, tr);
    CUIBM_TRY(cudaGetLastError());
}

template <int L>
static void split_table(Context &c, const double *src, int rows, int n, int nch, int ld_r, int ld_m,
                        const double *extra, __nv_bfloat16 *out, double *scale)
{
    if (nch * kKC <= 512)
        k_sep_split_table<L, 2><<<rows, 128, 0, c.stream>>>(src, n, nch, ld_r, ld_m, extra, out, scale);
    else
        k_sep_split_table<L, 8><<<rows, 128, 0, c.stream>>>(src, n, nch, ld_r, ld_m, extra, out, scale);
    CUIBM_TRY(cudaGetLastError());
}

static void launch_tri(Context &c, const SepPlan &P)
{
    const int nm = P.max_nm(), nr = P.max_nr();
    const int cb = tri_modes(nm, nr), threads = tri_threads(nm, nr), m = P.tri_rows;
    const dim3 grid((nm + cb - 1) / cb, P.grids);
    auto go = [&](auto *fn, size_t smem) { fn<<<grid, threads, smem, c.stream>>>(P.a, m); };
    const size_t rows = (size_t)m * kTriThreads * sizeof(double);
    if (cb == 8) {  // (600 modes and as many rows at least: ten rows a thread and more)
        if (m <= 16) go(k_sep_tri<8, 16, kTriThreads>, 0);
        else go(k_sep_tri<8, 0, kTriThreads>, rows);
    } else if (threads == 128) {
        if (m <= 2) go(k_sep_tri<4, 2, 128>, 0);
        else if (m <= 4) go(k_sep_tri<4, 4, 128>, 0);
        else if (m <= 6) go(k_sep_tri<4, 6, 128>, 0);
        else if (m <= 9) go(k_sep_tri<4, 9, 128>, 0);
        else if (m <= 12) go(k_sep_tri<4, 12, 128>, 0);
        else go(k_sep_tri<4, 16, 128>, 0);
    } else if (threads == 256) {
        if (m <= 12) go(k_sep_tri<4, 12, 256>, 0);
        else go(k_sep_tri<4, 16, 256>, 0);
    } else {
        go(k_sep_tri<4, 0, kTriThreads>, rows);
    }
    CUIBM_TRY(cudaGetLastError());
}

template <int L>
static void apply_t(Context &c, const SepPlan &P, const double *in, double *out, int tr)
{
    if (in) launch_split<L, false>(c, P, in, tr);  // (null: the digits are there already)
    if (in) stamp(c);  // digits of the field
    launch_gemm<L>(c, P, nullptr, 0);
    stamp(c);  // product with Q
    launch_tri(c, P);
    stamp(c);  // tridiagonal solves
    launch_split<L, true>(c, P, nullptr);
    stamp(c);  // digits of z^, pinned cells
    launch_gemm<L>(c, P, out, 1 + tr);
    stamp(c);  // product with Q^T
}

static void apply_grid(Context &c, const SepPlan &P, const double *in, double *out, int transposed = 0)
{
    if (P.digits == kDigits) apply_t<kDigits>(c, P, in, out, transposed);
    else apply_t<kDigitsMixed>(c, P, in, out, transposed);
}

// ---- rows that a body patches -----------------------------------------------------------
// With A = A0 + E P (E the m patched rows' unit vectors, P what those rows add to A0's),
// A^-1 r = A0^-1 (r - E q) where (I + P A0^-1 E) q = P A0^-1 r.  The m x m capacitance matrix
// is inverted once, at set-up, for a body whose rows stay; an application then is two of
// A0^-1 and a dense m x m product.
struct RowGap {  // (P y)_k at the patched row i: its row less the row that A0 has there
    Lhs1Coef full1, plain1;
    Lhs2Coef full, plain;
    Grid g;
    int which;
    __device__ double at(int i, const double *__restrict__ y) const
    {
        if (which == 1) return lhs1_row(full1, g, i, y) - lhs1_row(plain1, g, i, y);
        return lhs2_row(full, g, i, y) - lhs2_row(plain, g, i, y);
    }
};
static RowGap row_gap(const Context &c, int which)
{
    RowGap A{c.l1, c.l1, c.l2, c.l2, c.g, which};
    A.plain1.patch = A.plain.patch = RowPatch{};
    return A;
}
__global__ void k_sep_gap(RowGap A, int m, const int *__restrict__ row, const double *__restrict__ y, double *gap)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < m) gap[k] = A.at(row[k], y);
}

// q = cap gap, a warp a row
__global__ void k_sep_cap(int m, const double *__restrict__ cap, const double *__restrict__ gap, double *q)
{
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= m) return;
    double v = 0;
#pragma unroll 4
    for (int j = lane; j < m; j += 32) v += cap[(size_t)k * m + j] * gap[j];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) q[k] = v;
}

__global__ void k_sep_less(int n, const double *__restrict__ in, const int *__restrict__ idx,
                           const double *__restrict__ q, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i] - (idx[i] >= 0 ? q[idx[i]] : 0.0);
}

// set-up: a unit vector at cell `at`, the one before it cleared; a column of the capacitance
// matrix beside the identity; Gauss-Jordan with row exchanges on [m][2 m]
__global__ void k_sep_unit(double *v, int before, int at)
{
    if (before >= 0) v[before] = 0;
    v[at] = 1;
}
__global__ void k_sep_column(int m, int j, const double *__restrict__ gap, double *W)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    W[(size_t)k * 2 * m + j] = gap[k] + (k == j ? 1.0 : 0.0);
    W[(size_t)k * 2 * m + m + j] = k == j ? 1.0 : 0.0;
}
__global__ void __launch_bounds__(256) k_sep_pivot(int m, int k, double *W, double *fac, int *bad)
{
    __shared__ double big[256];
    __shared__ int who[256];
    double v = -1;
    int p = k;
    for (int i = k + threadIdx.x; i < m; i += 256) {
        const double a = fabs(W[(size_t)i * 2 * m + k]);
        if (a > v) v = a, p = i;
    }
    big[threadIdx.x] = v;
    who[threadIdx.x] = p;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o && big[threadIdx.x + o] > big[threadIdx.x]) {
            big[threadIdx.x] = big[threadIdx.x + o];
            who[threadIdx.x] = who[threadIdx.x + o];
        }
        __syncthreads();
    }
    p = who[0];
    const double piv = W[(size_t)p * 2 * m + k];
    __syncthreads();
    if (!(fabs(piv) > 1e-300)) {  // zero or not a number
        if (threadIdx.x == 0) *bad = 1;
        return;
    }
    for (int j = threadIdx.x; j < 2 * m; j += 256) {
        const double a = W[(size_t)p * 2 * m + j];
        if (p != k) W[(size_t)p * 2 * m + j] = W[(size_t)k * 2 * m + j];
        W[(size_t)k * 2 * m + j] = a / piv;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += 256) fac[i] = i == k ? 0.0 : W[(size_t)i * 2 * m + k];
}
__global__ void k_sep_eliminate(int m, int k, double *W, const double *__restrict__ fac)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j < 2 * m && i != k) W[(size_t)i * 2 * m + j] -= fac[i] * W[(size_t)k * 2 * m + j];
}

// A moving body's rows change every step, so nothing of theirs is inverted ahead.  Scaled to
// A0's diagonal before A0^-1 and swept once by Jacobi after it, z = y + D^-1 (r - A y) on the
// patched rows, they leave 8 to 11 iterations (embedded cylinder, 186 patched rows of 96100:
// 29 without either, 16 with the scaling alone; exact local solves of the rows' region: 10).
__global__ void k_sep_sweep(StoredOp2 A, int n, const double *__restrict__ r, const double *__restrict__ z, double *dz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int k = A.c.patch.pid[i];
    if (k < 0) return;
    const double own = A.c.patch.pdiag[k];
    dz[i] = own != 0 ? (r[i] - A.row(i, PtrAccess{z})) / own : 0.0;
}
__global__ void k_sep_add(int n, const int *__restrict__ pid, const double *__restrict__ dz, double *z)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && pid[i] >= 0) z[i] += dz[i];
}
// the transposed form: y = D^-1 r on the patched rows, then z = y + S A0^-T (r - A^T y)
__global__ void k_sep_first(RowPatch P, int n, const double *__restrict__ r, double *y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int k = P.pid[i];
    const double own = k >= 0 ? P.pdiag[k] : 0.0;
    y[i] = own != 0 ? r[i] / own : 0.0;
}
__global__ void k_sep_residual(Op2T A, int n, const double *__restrict__ r, const double *__restrict__ y, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = r[i] - A.row(i, PtrAccess{y});
}
__global__ void k_sep_last(const __grid_constant__ SepArgs args, int n, const double *__restrict__ y, double *z)
{
    const SepDev &d = args.f[0];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int k = d.patch.pid[i];
    if (k >= 0) z[i] = y[i] + z[i] * row_ratio(d, i, k);
}

// patched rows: the capacitance matrix is 8 m^2 bytes and its set-up m applications (a velocity
// system's twice the work of a pressure system's, against fewer iterations saved)
static int patch_max(int which) { return which == 1 ? 1024 : 2048; }

// out = M in: five kernels, or thirteen with patched rows
void launch_separable_apply(Context &c, LinearSystem &S, const double *in, double *out, bool digits)
{
    const SepPlan &P = *static_cast<const SepPlan *>(S.sep);
    if (P.moving) {
        apply_grid(c, P, in, out);
        const StoredOp2 A{c.l2, S.diag, nullptr, c.g.nx, c.g.ny};
        k_sep_sweep<<<blocks_for(S.n), kBlock, 0, c.stream>>>(A, S.n, in, out, P.y);
        k_sep_add<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, c.l2.patch.pid, P.y, out);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // sweep on the body's rows
        return;
    }
    if (!P.patched) {
        apply_grid(c, P, digits ? nullptr : in, out);
        return;
    }
    apply_grid(c, P, digits ? nullptr : in, P.y);
    const RowGap A = row_gap(c, S.which);
    k_sep_gap<<<blocks_for(P.patched), kBlock, 0, c.stream>>>(A, P.patched, P.prow, P.y, P.gap);
    k_sep_cap<<<blocks_for(32L * P.patched), kBlock, 0, c.stream>>>(P.patched, P.cap, P.gap, P.q);
    k_sep_less<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, in, P.pidx, P.q, P.rin);
    CUIBM_TRY(cudaGetLastError());
    stamp(c);  // capacitance of the body's rows
    apply_grid(c, P, P.rin, out);
}

// out = M^T in for the transposed solves of the embedded method's adjoint
void launch_separable_transposed(Context &c, LinearSystem &S, const TransposeList &T, const double *in, double *out)
{
    const SepPlan &P = *static_cast<const SepPlan *>(S.sep);
    const int n = S.n, nb = blocks_for(n);
    k_sep_first<<<nb, kBlock, 0, c.stream>>>(c.l2.patch, n, in, P.y);
    k_sep_residual<<<nb, kBlock, 0, c.stream>>>(Op2T{c.l2, c.g, T}, n, in, P.y, P.rin);
    CUIBM_TRY(cudaGetLastError());
    apply_grid(c, P, P.rin, out, 1);
    k_sep_last<<<nb, kBlock, 0, c.stream>>>(P.a, n, P.y, out);
    CUIBM_TRY(cudaGetLastError());
}

static char *plan_malloc(size_t bytes);

// The capacitance matrix of a fixed body's patched rows and its inverse.  False where it
// cannot be inverted or the body has too many rows for it.
static bool build_patch(Context &c, LinearSystem &S, const std::vector<int> &pid)
{
    SepPlan &P = *static_cast<SepPlan *>(S.sep);
    std::vector<int> rows, idx(S.n, -1);
    for (int i = 0; i < S.n; ++i)
        if (pid[i] >= 0) {
            idx[i] = (int)rows.size();
            rows.push_back(i);
        }
    const int m = (int)rows.size();
    if (m == 0) return true;
    if (m > patch_max(S.which)) return false;
    const size_t n = S.n, w = (size_t)2 * m * m;
    const size_t bytes = (2 * n + (size_t)m * m + 2 * (size_t)m) * 8 + (n + (size_t)m) * 4;
    P.pblock = plan_malloc(bytes);
    P.y = reinterpret_cast<double *>(P.pblock);
    P.rin = P.y + n;
    P.cap = P.rin + n;
    P.gap = P.cap + (size_t)m * m;
    P.q = P.gap + m;
    P.pidx = reinterpret_cast<int *>(P.q + m);
    P.prow = P.pidx + n;
    CUIBM_TRY(cudaMemcpyAsync(P.pidx, idx.data(), n * 4, cudaMemcpyHostToDevice, c.stream));
    CUIBM_TRY(cudaMemcpyAsync(P.prow, rows.data(), m * 4, cudaMemcpyHostToDevice, c.stream));
    char *tmp = plan_malloc((w + m) * 8 + 256);
    struct Freed {
        char *p;
        ~Freed() { cudaFree(p); }
    } freed{tmp};
    double *W = reinterpret_cast<double *>(tmp), *fac = W + w;
    int *bad = reinterpret_cast<int *>(fac + m), hbad = 0;
    CUIBM_TRY(cudaMemsetAsync(bad, 0, 4, c.stream));
    CUIBM_TRY(cudaMemsetAsync(P.rin, 0, n * 8, c.stream));
    const RowGap A = row_gap(c, S.which);
    for (int j = 0; j < m; ++j) {
        k_sep_unit<<<1, 1, 0, c.stream>>>(P.rin, j ? rows[j - 1] : -1, rows[j]);
        apply_grid(c, P, P.rin, P.y);
        k_sep_gap<<<blocks_for(m), kBlock, 0, c.stream>>>(A, m, P.prow, P.y, P.gap);
        k_sep_column<<<blocks_for(m), kBlock, 0, c.stream>>>(m, j, P.gap, W);
    }
    for (int k = 0; k < m; ++k) {
        k_sep_pivot<<<1, 256, 0, c.stream>>>(m, k, W, fac, bad);
        k_sep_eliminate<<<dim3(blocks_for(2L * m), m), kBlock, 0, c.stream>>>(m, k, W, fac);
    }
    CUIBM_TRY(cudaGetLastError());
    CUIBM_TRY(cudaMemcpy2DAsync(P.cap, (size_t)m * 8, W + m, (size_t)2 * m * 8, (size_t)m * 8, m,
                                cudaMemcpyDeviceToDevice, c.stream));
    CUIBM_TRY(cudaMemcpyAsync(&hbad, bad, 4, cudaMemcpyDeviceToHost, c.stream));
    CUIBM_TRY(cudaStreamSynchronize(c.stream));
    P.patched = m;
    return !hbad;
}

// Where the separable preconditioner takes the place of the smoothed-aggregation cycle: the
// pressure system of the methods that leave its rows alone, unless the case asks for a form
// of smoothed aggregation by name (-saStructured 0 or 1, strengthThreshold, -separable 0).
// By itself (-separable -1) not where the pressure's level would move by more than 1e-9 of
// it: with the external and embedded methods one pinned cell in the domain's corner fixes the level, and
// the smoothed-aggregation solves leave their stopping error in it (against a solve to
// 1e-15: 1e-10 to 1e-7 of p at a relative residual of 1e-13 from 200k unknowns on, 1e-9 in
// mixed precision and in batches at 1e-12, below 3e-10 elsewhere; the separable solves
// 1e-11; embedded, 470k unknowns at 1e-12: up to 1.0e-9 against 4e-10), so runs there keep
// the solver that they began with unless they ask (-separable 1: Re 550, 922 x 922, 101 to
// 2.8 ms a step, the oscillating cylinder 686 x 686 34.5 to 10.1 ms).  With the plain and
// Fadlun methods the centre cell is pinned too and the level agrees to 1e-10.
constexpr int kLevelMax = 200000;

// The velocity system (I - dt/2 nu L, two grids) has a far smaller condition number, and the
// diagonally preconditioned iteration is good where it needs few steps.  Its matrix D^-1 A
// has its spectrum in 1 +- s / (1 + s), s the largest sum of a row's coefficients, so a
// BiCGSTAB step (two products) gains ((sqrt(1 + 2 s) - 1) / (sqrt(1 + 2 s) + 1))^2; the
// prediction is 1.2 to 1.3 times the measured count (Re 40: 18 against 14, Re 550: 9
// against 7).
static double predicted_velocity_steps(const Context &c, double rtol)
{
    const double *t = c.htab.data();
    const int nx = c.g.nx, ny = c.g.ny;
    auto largest = [&](const char *a, const char *b, int n) {
        double m = 0;
        for (int i = 0; i < n; ++i) m = std::max(m, t[c.hoff.at(a) + i] + t[c.hoff.at(b) + i]);
        return m;
    };
    const double s = std::max(largest("1uE", "1uW", nx - 1) + largest("1uN", "1uS", ny),
                              largest("1vE", "1vW", nx) + largest("1vN", "1vS", ny - 1));
    const double q = (std::sqrt(1 + 2 * s) - 1) / (std::sqrt(1 + 2 * s) + 1);
    return q > 0 ? std::log(2 / rtol) / (2 * std::log(1 / q)) : 0.0;
}
// From this predicted count on (FP64, one application against n steps of the diagonal one: 64 x
// 64 70 us against 97 at 3.8 and 124 at 5.2, 270 x 270 122 against 115 and 146, 512 x 512 218
// against 191 and 247; 900 x 900 745 against 662 at 5.2 and 819 at 6.6)
static double velocity_steps(const LinearSystem &S) { return S.n > 600000 ? 6.5 : 5; }

static bool separable_applies(const Context &c, const LinearSystem &S)
{
    const int nx = c.g.nx, ny = c.g.ny;
    if (c.P.separable == 0 || std::min(nx, ny) > kSepMax || std::max(nx, ny) > kTriRows) return false;
    if (S.which == 2) {
        if (S.precond != PC_SMOOTHED_AGGREGATION || c.P.saStructured != -1 || c.P.poisson.strength >= 0) return false;
    } else {
        if (S.precond != PC_DIAGONAL || c.P.solverType == ST_OSC) return false;
    }
    if (c.P.separable == 1) return true;
    const bool level = c.P.solverType == ST_NAVIERSTOKES || c.P.solverType == ST_FADLUN ||
                       (c.g.nP < kLevelMax && c.P.solverPack != 2 &&
                        c.P.poisson.precision == PRECISION_FP64);
    // a pressure system of one level is solved by its dense inverse in one launch: 10 to 20 us less
    // than this chain up to 1444 unknowns, bodies 10 to 490 us (a moving one's rows are exact there);
    // at 1600, with two levels, the step takes 103 us here against 133 (1e-5) to 537 (1e-12)
    return level && (S.which == 2 ? c.g.nP > kCoarse : predicted_velocity_steps(c, S.rtol) >= velocity_steps(S));
}

// One grid's operator: shift + X + Y with the coefficients towards the next and the
// previous node (um, dm along the transform, ur, dr along the rows; all of them in the
// diagonal) and the weights that make X symmetric (wm; wr with them the rows of CG's system)
struct SepGrid {
    double shift;
    std::vector<double> um, dm, wm, ur, dr, wr;
    int sm, sr, base;
    std::vector<int> pin_m, pin_r;
};

// Device memory for the plan.  A context that does not get it keeps its smoothed-aggregation
// or diagonal preconditioner (NoRoom, caught in setup_separable) instead of failing.
struct NoRoom {};
static char *plan_malloc(size_t bytes)
{
    void *p = nullptr;
    const cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw NoRoom{};
    }
    CUIBM_TRY(e);
    return static_cast<char *>(p);
}

// The tables of grid g into P.a.f[g]; false where the eigenvalues do not converge or the pinned
// cells' correction is singular: the system then keeps its other preconditioner.  nq: the threads
// a mode of k_sep_tri (the same for all grids of a launch).
static bool build_grid(Context &c, SepPlan &P, int g, const SepGrid &G, bool sym, int nq)
{
    SepDev &d = P.a.f[g];
    const int L = P.digits, nm = (int)G.um.size(), nr = (int)G.ur.size();
    d.nm = nm;
    d.nr = nr;
    d.sm = G.sm;
    d.sr = G.sr;
    d.base = G.base;
    d.nch = (nm + kKC - 1) / kKC;
    d.pins = (int)G.pin_m.size();
    // eigenvalues of D^1/2 X D^-1/2 and the rotations that give its eigenvectors
    std::vector<double> lam(nm), off(nm, 0.0);
    for (int i = 0; i < nm; ++i) lam[i] = G.um[i] + G.dm[i];
    for (int i = 0; i + 1 < nm; ++i) off[i] = -std::sqrt(G.um[i] * G.dm[i + 1]);
    std::vector<Sweep> sweeps;
    std::vector<double2> rot;
    if (!tridiagonal_qr(lam, off, sweeps, rot)) return false;
    // a system with pinned cells is singular without them: the constant is exactly X's null vector
    const int k0 = d.pins ? (int)(std::min_element(lam.begin(), lam.end()) - lam.begin()) : -1;
    if (d.pins) lam[k0] = 0;
    double len = 0;
    for (double w : G.wm) len += w;
    std::vector<double> cm(nm), cr(nr), em(nm), con(nm), et(nm), crt(nr);
    for (int J = 0; J < nr; ++J) crt[J] = 1 / G.wr[J];
    for (int i = 0; i < nm; ++i) {
        et[i] = std::sqrt(G.wm[i]);
        cm[i] = sym ? 1 / std::sqrt(G.wm[i]) : std::sqrt(G.wm[i]);
        em[i] = 1 / std::sqrt(G.wm[i]);
        con[i] = std::sqrt(G.wm[i] / len);
    }
    for (int J = 0; J < nr; ++J) cr[J] = sym ? 1 / G.wr[J] : 1.0;

    // one allocation for all tables and work arrays
    const size_t n = (size_t)nm * nr, dig = (size_t)d.nch * L * kKC;
    size_t need = 0;
    auto reserve = [&](size_t bytes) {
        const size_t at = need;
        need += (bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t oB1 = reserve(nm * dig * 2), oB2 = reserve(nm * dig * 2), oA = reserve(nr * dig * 2);
    const size_t osB1 = reserve(nm * 8), osB2 = reserve(nm * 8), osA = reserve(nr * 8);
    const size_t oh = reserve(n * 8), ol = reserve(n * 8), oc = reserve(n * 8), oi = reserve(n * 8);
    const size_t oPf = reserve((size_t)nq * nm * 8), oPb = reserve((size_t)nq * nm * 8);
    const size_t ocmt = reserve(nm * 8), ocrt = reserve(nr * 8), osB2t = reserve(nm * 8), owr = reserve(nr * 8);
    const size_t ocm = reserve(nm * 8), ocr = reserve(nr * 8), oF0 = reserve(nm * 8), oF1 = reserve(nm * 8);
    const size_t oG0 = reserve(d.pins > 0 ? n * 8 : 8), oG1 = reserve(d.pins > 1 ? n * 8 : 8), ogm = reserve(nr * 8);
    P.block[g] = plan_malloc(need);
    char *block = P.block[g];
    auto D = [&](size_t at) { return reinterpret_cast<double *>(block + at); };
    auto H = [&](size_t at) { return reinterpret_cast<__nv_bfloat16 *>(block + at); };
    auto put = [&](double *dst, const std::vector<double> &v) {
        CUIBM_TRY(cudaMemcpyAsync(dst, v.data(), v.size() * 8, cudaMemcpyHostToDevice, c.stream));
    };
    // set-up scratch, freed at the end
    const size_t bq = ((size_t)nm * nm * 8 + 255) & ~size_t(255), bs = (sweeps.size() * sizeof(Sweep) + 511) & ~size_t(255),
                 br = (rot.size() * sizeof(double2) + 511) & ~size_t(255), bv = (size_t)(4 * nm + 2 * nr) * 8;
    char *tmp = plan_malloc(bq + bs + br + bv);
    struct Freed {
        char *p;
        ~Freed() { cudaFree(p); }
    } freed{tmp};
    double *Q = reinterpret_cast<double *>(tmp);
    Sweep *sw = reinterpret_cast<Sweep *>(tmp + bq);
    double2 *rt = reinterpret_cast<double2 *>(tmp + bq + bs);
    double *vl = reinterpret_cast<double *>(tmp + bq + bs + br), *vcon = vl + nm, *vem = vcon + nm, *vet = vem + nm,
           *vur = vet + nm, *vdr = vur + nr;
    if (!rot.empty()) {
        CUIBM_TRY(cudaMemcpyAsync(sw, sweeps.data(), sweeps.size() * sizeof(Sweep), cudaMemcpyHostToDevice, c.stream));
        CUIBM_TRY(cudaMemcpyAsync(rt, rot.data(), rot.size() * sizeof(double2), cudaMemcpyHostToDevice, c.stream));
    }
    put(vl, lam);
    put(vcon, con);
    put(vem, em);
    put(vur, G.ur);
    put(vdr, G.dr);
    put(D(ocm), cm);
    put(D(ocr), cr);
    put(vet, et);
    put(D(ocmt), em);
    put(D(ocrt), crt);
    put(D(owr), G.wr);
    const size_t smem = (size_t)nm * kRotWarps * 8;
    allow_smem(k_sep_rotate, (size_t)kSepMax * kRotWarps * 8);
    k_sep_rotate<<<(nm + kRotWarps - 1) / kRotWarps, 32 * kRotWarps, smem, c.stream>>>(nm, sw, (int)sweeps.size(), rt, Q);
    if (d.pins) k_sep_constant<<<blocks_for(nm), kBlock, 0, c.stream>>>(nm, k0, vcon, Q);
    CUIBM_TRY(cudaGetLastError());
    if (L == kDigits) {
        allow_gemm<kDigits>();
        split_table<kDigits>(c, Q, nm, nm, d.nch, 1, nm, nullptr, H(oB1), D(osB1));
        split_table<kDigits>(c, Q, nm, nm, d.nch, nm, 1, vet, H(oB2), D(osB2t));
        split_table<kDigits>(c, Q, nm, nm, d.nch, nm, 1, vem, H(oB2), D(osB2));
    } else {
        allow_gemm<kDigitsMixed>();
        split_table<kDigitsMixed>(c, Q, nm, nm, d.nch, 1, nm, nullptr, H(oB1), D(osB1));
        split_table<kDigitsMixed>(c, Q, nm, nm, d.nch, nm, 1, vet, H(oB2), D(osB2t));
        split_table<kDigitsMixed>(c, Q, nm, nm, d.nch, nm, 1, vem, H(oB2), D(osB2));
    }
    allow_smem(k_sep_tri<8, 0, kTriThreads>, 200 * 1024);
    allow_smem(k_sep_tri<4, 0, kTriThreads>, 200 * 1024);
    const double reg = d.pins ? G.ur[0] : 0.0;
    k_sep_factor<<<(nm + 31) / 32, 32, 0, c.stream>>>(nm, nr, nq, P.tri_rows, vur, vdr, vl, G.shift, k0, reg, D(ol), D(oc),
                                                      D(oi), D(oPf), D(oPb));
    CUIBM_TRY(cudaGetLastError());
    d.B1 = H(oB1);
    d.B2 = H(oB2);
    d.A = H(oA);
    d.sB1 = D(osB1);
    d.sB2 = D(osB2);
    d.sA = D(osA);
    d.h = D(oh);
    d.l = D(ol);
    d.c = D(oc);
    d.inv = D(oi);
    d.Pf = D(oPf);
    d.Pb = D(oPb);
    d.cm = D(ocm);
    d.cr = sym ? D(ocr) : nullptr;
    d.cmt = D(ocmt);
    d.crt = D(ocrt);
    d.sB2t = D(osB2t);
    d.wr = D(owr);
    d.k0 = k0;
    d.mean = 1 / std::sqrt(len);
    d.gm = D(ogm);
    CUIBM_TRY(cudaStreamSynchronize(c.stream));
    if (!d.pins) return true;

    // Pinned cells and the constant.  With B = A0 plus reg on the constant's mode in row 0,
    // A = B + sum_p delta_p e_p e_p^T - reg u mean^T (u one on row 0, mean the average over
    // it), so z = B^-1 r - sum_p q_p G_p + q_m G_m with q_p = delta_p z_p, q_m = reg mean(z)
    const int np = d.pins;
    std::vector<std::vector<double>> F(2, std::vector<double>(nm));
    std::vector<double> row(nm);
    double *Gp[2] = {D(oG0), D(oG1)}, *Fp[2] = {D(oF0), D(oF1)};
    double delta[2] = {0, 0}, at_pin[3][3] = {};  // functional a of response b
    for (int p = 0; p < np; ++p) {
        const int m = G.pin_m[p], R = G.pin_r[p];
        delta[p] = G.um[m] + G.dm[m] + G.ur[R] + G.dr[R];
        CUIBM_TRY(cudaMemcpyAsync(row.data(), Q + (size_t)m * nm, nm * 8, cudaMemcpyDeviceToHost, c.stream));
        CUIBM_TRY(cudaStreamSynchronize(c.stream));
        for (int k = 0; k < nm; ++k) F[p][k] = row[k] * em[m];
        for (int k = 0; k < nm; ++k) row[k] *= std::sqrt(G.wm[m]);
        put(Fp[p], F[p]);
        CUIBM_TRY(cudaMemsetAsync(d.h, 0, n * 8, c.stream));
        put(d.h + (size_t)R * nm, row);
        launch_tri(c, P);
        CUIBM_TRY(cudaMemcpyAsync(Gp[p], d.h, n * 8, cudaMemcpyDeviceToDevice, c.stream));
        CUIBM_TRY(cudaStreamSynchronize(c.stream));
        d.R[p] = R;
        d.F[p] = Fp[p];
        d.G[p] = Gp[p];
    }
    // the constant's response: mode k0 only, u = sqrt(len) there
    CUIBM_TRY(cudaMemsetAsync(d.h, 0, n * 8, c.stream));
    put(d.h + k0, std::vector<double>(1, std::sqrt(len)));
    launch_tri(c, P);
    CUIBM_TRY(cudaMemcpy2DAsync(D(ogm), 8, d.h + k0, (size_t)nm * 8, 8, nr, cudaMemcpyDeviceToDevice, c.stream));
    for (int b = 0; b <= np; ++b) {  // responses: the pins', then the constant's
        const double *src = b < np ? Gp[b] : d.h;
        for (int a = 0; a <= np; ++a) {
            CUIBM_TRY(cudaMemcpyAsync(row.data(), src + (size_t)(a < np ? d.R[a] : 0) * nm, nm * 8,
                                      cudaMemcpyDeviceToHost, c.stream));
            CUIBM_TRY(cudaStreamSynchronize(c.stream));
            double v = 0;
            if (a < np)
                for (int k = 0; k < nm; ++k) v += F[a][k] * row[k];
            else
                v = row[k0] * d.mean;
            at_pin[a][b] = v;
        }
    }
    for (int a = 0; a <= np; ++a)
        for (int b = 0; b <= np; ++b) d.K[3 * a + b] = b == np ? -at_pin[a][b] : at_pin[a][b];
    for (int p = 0; p < np; ++p) d.K[3 * p + p] += 1 / delta[p];
    d.K[3 * np + np] += 1 / reg;
    return invert3(d.K, np + 1);
}

static void build_separable(Context &c, LinearSystem &S);

void setup_separable(Context &c, LinearSystem &S)
{
    try {
        build_separable(c, S);
    } catch (const NoRoom &) {
        CUIBM_TRY(cudaStreamSynchronize(c.stream));
        free_separable(S);
    }
}

static void build_separable(Context &c, LinearSystem &S)
{
    ++S.tables;
    S.sep = nullptr;
    if (!separable_applies(c, S) || !S.diag) return;  // (the stored diagonal comes with the persistent solver)
    const int nx = c.g.nx, ny = c.g.ny;
    const bool alongx = nx <= ny;  // the shorter direction is transformed: n_m^2 n_r work
    const double *t = c.htab.data();
    auto tab = [&](const char *k, int n) { return std::vector<double>(t + c.hoff.at(k), t + c.hoff.at(k) + n); };
    const std::vector<double> &dx = c.gx.width, &dy = c.gy.width;
    auto between = [](const std::vector<double> &w) {  // face nodes
        std::vector<double> f(w.size() - 1);
        for (size_t i = 0; i < f.size(); ++i) f[i] = 0.5 * (w[i] + w[i + 1]);
        return f;
    };
    std::vector<SepGrid> grids;
    auto add = [&](double shift, int mx, int my, int base, const char *e, const char *w, const char *n, const char *s,
                   const std::vector<double> &wx, const std::vector<double> &wy) {
        SepGrid G;
        G.shift = shift;
        G.base = base;
        G.sm = alongx ? 1 : mx;
        G.sr = alongx ? mx : 1;
        G.um = alongx ? tab(e, mx) : tab(n, my);
        G.dm = alongx ? tab(w, mx) : tab(s, my);
        G.ur = alongx ? tab(n, my) : tab(e, mx);
        G.dr = alongx ? tab(s, my) : tab(w, mx);
        G.wm = alongx ? wx : wy;
        G.wr = alongx ? wy : wx;
        grids.push_back(G);
    };
    if (S.which == 1) {
        add(1.0, nx - 1, ny, 0, "1uE", "1uW", "1uN", "1uS", between(dx), dy);
        add(1.0, nx, ny - 1, c.g.nU, "1vE", "1vW", "1vN", "1vS", dx, between(dy));
    } else {
        add(0.0, nx, ny, 0, "2E", "2W", "2N", "2S", dx, dy);
        for (int cell : {c.l2.pin0, c.l2.pinc}) {
            if (cell < 0) continue;
            grids[0].pin_m.push_back(alongx ? cell % nx : cell / nx);
            grids[0].pin_r.push_back(alongx ? cell / nx : cell % nx);
        }
    }
    SepPlan *P = new SepPlan();
    S.sep = P;
    P->digits = S.precision == PRECISION_MIXED && c.P.solverType == ST_FADLUN ? kDigitsMixed : kDigits;
    int nm = 0, nr = 0;
    for (const SepGrid &G : grids) {
        nm = std::max(nm, (int)G.um.size());
        nr = std::max(nr, (int)G.ur.size());
    }
    const int nq = tri_threads(nm, nr) / tri_modes(nm, nr);
    P->tri_rows = (nr + nq - 1) / nq;
    for (size_t g = 0; g < grids.size(); ++g) {
        P->grids = 1;
        if (!build_grid(c, *P, (int)g, grids[g], S.w != nullptr, nq)) {
            free_separable(S);
            return;
        }
    }
    P->grids = (int)grids.size();
    // the row kernels: contiguous rows, of an operator whose rows stay (64 x 64 cavity step 220
    // -> 205 us, 270 x 270 cylinder 442 -> 437, 512 x 512 mixed 753 -> 762: there the vector
    // kernels are bound by bandwidth and the flat ones are the better)
    P->rows = alongx && nm <= kRowPlaces && !(S.which == 2 && c.P.solverType == ST_OSC);
    P->sums_cap = std::max(kRowBlocks, nr * P->grids);
    const size_t sums = (6 * (size_t)P->sums_cap + 2) * sizeof(double);
    P->sums = reinterpret_cast<double *>(plan_malloc(sums));
    CUIBM_TRY(cudaMemsetAsync(P->sums, 0, sums, c.stream));
    if (!(S.which == 1 ? c.l1.patch.pid : c.l2.patch.pid)) return;
    if (c.P.solverType == ST_OSC) {
        SepDev &d = P->a.f[0];
        d.patch = c.l2.patch;
        d.E = c.l2.E;
        d.W = c.l2.W;
        d.N = c.l2.N;
        d.S = c.l2.S;
        d.nx = nx;
        P->moving = true;
        P->pblock = plan_malloc(2 * (size_t)S.n * sizeof(double));
        P->y = reinterpret_cast<double *>(P->pblock);
        P->rin = P->y + S.n;
    } else if (!build_patch(c, S, S.which == 1 ? c.fadlun.pid1 : c.fadlun.pid2)) {
        free_separable(S);
    }
}

void free_separable(LinearSystem &S)
{
    SepPlan *P = static_cast<SepPlan *>(S.sep);
    if (!P) return;
    if (P->pblock) cudaFree(P->pblock);
    if (P->sums) cudaFree(P->sums);
    for (char *b : P->block)
        if (b) cudaFree(b);
    delete P;
    S.sep = nullptr;
    ++S.tables;
}

// ---- host side: solves --------------------------------------------------------------------
namespace {

struct SepSolve {
    Context &c;
    LinearSystem &S;
    const double *b;
    double *x;

    template <class F>
    void with_op(const F &f) const
    {
        if (S.which == 1) f(StoredOp1{c.l1, S.diag, S.w, c.g.nx, c.g.ny, c.g.nU});
        else f(StoredOp2{c.l2, S.diag, S.w, c.g.nx, c.g.ny});
    }
    int nb() const { return row_blocks(S.n); }
    SepPlan &plan() const { return *static_cast<SepPlan *>(S.sep); }
    // the launches while it lives are the first application's and look at the gate
    struct Gated {
        SepGate &gate;
        Gated(const SepSolve &L, bool first) : gate(L.plan().a.gate)
        {
            const SepPlan &P = L.plan();
            if (!first) return;
            if (!P.rows) {
                gate.status = &L.S.ks->status;
            } else if (L.S.rtol > 1e-140 && L.S.rtol < 0.5) {  // (rtol^2 and its product with ||b||^2 in range)
                gate.acc = P.sums + 6 * (size_t)P.sums_cap;
                gate.m = 2 * (float)std::frexp(L.S.rtol * L.S.rtol, &gate.e);
                --gate.e;
            }
        }
        explicit Gated(const SepSolve &L, const int *skip) : gate(L.plan().a.gate) { gate.status = skip; }
        ~Gated() { gate = SepGate{}; }
    };
    RowSums sums() const
    {
        const SepPlan &P = plan();
        return RowSums{P.sums, P.sums_cap, P.max_nr() * P.grids, nb()};
    }
    // f(digits, pairs a thread) as compile-time constants, for the row kernels
    template <class F>
    void with_rows(const F &f) const
    {
        const SepPlan &P = plan();
        const int np = ((P.max_nm() + kKC - 1) / kKC * kKC + 255) / 256;
        auto pairs = [&](auto l) {
            if (np <= 1) f(l, std::integral_constant<int, 1>{});
            else f(l, std::integral_constant<int, 2>{});
        };
        if (P.digits == kDigits) pairs(std::integral_constant<int, kDigits>{});
        else pairs(std::integral_constant<int, kDigitsMixed>{});
    }
    dim3 row_grid() const { return dim3(plan().max_nr(), plan().grids); }

    // the first iteration by rows (k_row_*)
    template <bool CG>
    void row_start() const
    {
        with_op([&](auto A) {
            with_rows([&](auto l, auto np) {
                k_row_start<decltype(A), l(), np(), CG>
                    <<<row_grid(), 128, 0, c.stream>>>(plan().a, A, b, x, S.r, sums());
            });
        });
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // residual and its digits
    }
    void row_half(cudaGraphConditionalHandle h, int use) const
    {
        const Gated gated(*this, true);
        launch_separable_apply(c, S, S.r, S.Mp, true);
        with_op([&](auto A) {
            k_row_apply<decltype(A), 0>
                <<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.Mp, S.AMp, S.r, nullptr, sums(), 2);
        });
        stamp(c);  // A M r
        with_rows([&](auto l, auto np) {
            k_row_half<l(), np()><<<row_grid(), 128, 0, c.stream>>>(plan().a, S.r, S.AMp, S.Mp, S.s, x, sums(), S.ks,
                                                                     c.err_word, S.which, h, use);
        });
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // half step and its digits
    }
    void row_rest(cudaGraphConditionalHandle h, int use) const
    {
        launch_separable_apply(c, S, S.s, S.Ms, true);
        with_op([&](auto A) {
            k_row_apply<decltype(A), 1>
                <<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.Ms, S.AMs, S.s, nullptr, sums(), 2);
        });
        stamp(c);  // A M s
        k_row_end<<<nb(), kBlock, 0, c.stream>>>(S.n, x, S.r, S.rs, S.p, S.s, S.Ms, S.AMs, sums(), S.ks, c.err_word,
                                                 S.which, h, use);
        k_bicg_5<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.p, S.r, S.AMp, S.ks);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // end of the iteration, next direction
    }
    void row_cg(bool first, cudaGraphConditionalHandle h, int use) const
    {
        const Gated gated(*this, first);
        launch_separable_apply(c, S, S.r, S.z, true);
        with_op([&](auto A) {
            if (first) {
                k_row_apply<decltype(A), 2>
                    <<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.z, S.q, S.r, S.p, sums(), 2);
            } else {
                k_cg_rz<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.r, S.z, S.partials, S.ks);
                k_cg_3<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.p, S.z, S.ks);
                k_cg_1<<<blocks_for(S.n), kBlock, 0, c.stream>>>(A, S.n, S.p, S.q, S.partials, S.ks);
            }
        });
        stamp(c);  // direction and A p
        with_rows([&](auto l, auto np) {
            k_row_cg<l(), np()><<<row_grid(), 128, 0, c.stream>>>(plan().a, S.w, S.p, S.q, S.r, x, sums(), S.ks,
                                                                   c.err_word, S.which, first, h, use);
        });
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // CG step and the digits of r
    }

    void init() const
    {
        if (plan().rows) {
            if (S.krylov == KRYLOV_CG) row_start<true>();
            else row_start<false>();
            return;
        }
        with_op([&](auto A) {
            if (S.krylov == KRYLOV_CG)
                k_cg_init<decltype(A), 2><<<blocks_for(S.n), kBlock, 0, c.stream>>>(A, S.n, b, S.w, x, S.r, S.z, S.p, S.dinv,
                                                                        S.partials, S.ks, c.err_word, S.which, 0, 0);
            else
                k_sep_init<<<nb(), kBlock, 0, c.stream>>>(A, S.n, b, x, S.r, S.partials, S.ks, c.err_word, S.which);
        });
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // residual
    }
    // BiCGSTAB to the half step
    void half(bool first, cudaGraphConditionalHandle h, int use) const
    {
        if (first && plan().rows) {
            row_half(h, use);
            return;
        }
        const Gated gated(*this, first);
        launch_separable_apply(c, S, first ? S.r : S.p, S.Mp);
        with_op([&](auto A) {
            k_sep_1<<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.Mp, S.AMp, first ? S.r : S.rs, S.partials, S.ks, first);
        });
        stamp(c);  // A M p
        k_sep_2<<<nb(), kBlock, 0, c.stream>>>(S.n, S.r, S.AMp, S.Mp, S.s, x, S.partials, S.ks, first, h, use);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // half step
    }
    // and from there
    void rest(bool first, cudaGraphConditionalHandle h, int use) const
    {
        if (first && plan().rows) {
            row_rest(h, use);
            return;
        }
        launch_separable_apply(c, S, S.s, S.Ms);
        with_op([&](auto A) {
            k_sep_3<<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.s, S.Ms, S.AMs, S.partials, S.ks);
        });
        stamp(c);  // A M s, omega
        k_sep_4<<<nb(), kBlock, 0, c.stream>>>(S.n, x, S.r, S.rs, S.p, S.s, S.Ms, S.AMs, S.partials, S.ks, c.err_word,
                                               S.which, first, h, use);
        k_bicg_5<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.p, S.r, S.AMp, S.ks);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // end of the iteration and next direction
    }
    void correct() const
    {
        const int nb = blocks_for(S.n);
        const Gated gated(*this, &S.ks->skip);
        k_sep_pick<<<nb, kBlock, 0, c.stream>>>(S.n, S.r, S.s, S.p, S.ks);
        launch_separable_apply(c, S, S.p, S.Mp);
        with_op([&](auto A) { k_sep_accept<<<this->nb(), kBlock, 0, c.stream>>>(A, S.n, S.p, S.Mp, S.partials, S.ks); });
        k_sep_correct<<<nb, kBlock, 0, c.stream>>>(S.n, S.Mp, x, S.ks);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // last correction
    }
    void cg(bool first, cudaGraphConditionalHandle h, int use) const
    {
        if (plan().rows) {
            row_cg(first, h, use);
            return;
        }
        const Gated gated(*this, first);
        launch_separable_apply(c, S, S.r, S.z);
        with_op([&](auto A) {
            if (first) {
                k_sep_cg_1<<<nb(), kBlock, 0, c.stream>>>(A, S.n, S.r, S.z, S.p, S.q, S.partials, S.ks);
            } else {
                k_cg_rz<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.r, S.z, S.partials, S.ks);
                k_cg_3<<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, S.p, S.z, S.ks);
                k_cg_1<<<blocks_for(S.n), kBlock, 0, c.stream>>>(A, S.n, S.p, S.q, S.partials, S.ks);
            }
        });
        stamp(c);  // CG direction and A p
        k_cg_2<2><<<blocks_for(S.n), kBlock, 0, c.stream>>>(S.n, x, S.r, S.z, S.p, S.q, S.w, S.dinv, S.partials, S.ks, c.err_word,
                                                 S.which, h, use);
        CUIBM_TRY(cudaGetLastError());
        stamp(c);  // CG step
    }
};

}  // namespace

// A solve on c.stream.  Captured into the step's graph, the first half iteration (CG: the
// first iteration) is plain nodes, the rest of it an IF node and further iterations a WHILE
// node, both skipped by the solves that have converged; otherwise the host reads the
// status after each.
void launch_separable_solve(Context &c, LinearSystem &S, const double *b, double *x, bool in_graph)
{
    const SepSolve L{c, S, b, x};
    SepPlan &P = *static_cast<SepPlan *>(S.sep);
    const bool cg = S.krylov == KRYLOV_CG;
    const Traced traced(c, S.which);
    if (in_graph) {
        L.init();
        CondNode more(c);
        if (cg) {
            L.cg(true, more.h, 1);
            S.body_kernels = more.add(cudaGraphCondTypeWhile, [&] { L.cg(false, more.h, 1); });
            P.first_kernels = S.body_kernels;
            return;
        }
        CondNode second(c);
        L.half(true, second.h, 1);
        P.first_kernels = second.add(cudaGraphCondTypeIf, [&] { L.rest(true, more.h, 1); });
        S.body_kernels = more.add(cudaGraphCondTypeWhile, [&] {
            L.half(false, more.h, 1);
            L.rest(false, more.h, 1);
        });
        if (P.moving) L.correct();
        return;
    }
    KrylovScalars host{};
    auto running = [&] {
        CUIBM_TRY(cudaMemcpyAsync(&host, S.ks, sizeof(host), cudaMemcpyDeviceToHost, c.stream));
        CUIBM_TRY(cudaStreamSynchronize(c.stream));
        return host.status == KS_RUNNING;
    };
    L.init();
    if (cg) {
        L.cg(true, 0, 0);
        while (running()) L.cg(false, 0, 0);
        return;
    }
    L.half(true, 0, 0);
    for (bool first = true; running(); first = false) {
        if (!first) L.half(false, 0, 0);
        L.rest(first, 0, 0);
    }
    if (P.moving) L.correct();
}

// kernels that a solve's conditional bodies ran: the first execution is the rest of the
// first iteration, the later ones whole iterations
long long separable_body_launches(const LinearSystem &S, int runs)
{
    const SepPlan &P = *static_cast<const SepPlan *>(S.sep);
    return runs > 0 ? P.first_kernels + (long long)(runs - 1) * S.body_kernels : 0;
}

// Algorithmic bytes of a solve with `it` iterations: the residual, and for each application
// of the preconditioner its input, output, digits of one operand, the transform's two
// tables and the tridiagonal factors, with the operator applied to the result
double separable_bytes(const LinearSystem &S, int it)
{
    const SepPlan &P = *static_cast<const SepPlan *>(S.sep);
    const double n = S.n, nm = P.a.f[0].nm, L = P.digits;
    const double app = 8 * n * 2 + 2 * 2 * L * (n + nm * nm) + 8 * n * (2 + 3 + 2) + 8 * n * 5;
    const double apps = S.krylov == KRYLOV_CG ? std::max(it, 1) : 1 + 2 * std::max(0.0, it - 0.5);
    return 8 * n * 3 + apps * app;
}

}  // namespace cuibm
