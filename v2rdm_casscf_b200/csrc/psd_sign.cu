// PSD projection without an eigendecomposition: x = U+ / mu and z = U- from the
// matrix sign of U, by matrix products alone (FP64).
//
// With S = U scaled to norm <= 1, X <- a X - b X^3 (two products of symmetric
// matrices that commute) drives every eigenvalue of X from that of S towards
// its sign.  "Lift" steps take the cubic with the largest slope at 0 that
// keeps [0, 1] in [0, 1] and 1 above 0.246: each multiplies small eigenvalues by
// 2.46.  Then six "finish" steps, the equal-ripple cubics from [0.246, 1] on,
// take every lifted eigenvalue to +-1 to rounding (the last are Newton-Schulz
// steps).  Y = S X = |S| and Q = Y X give D = S - Q = S (1 - X^2), whose norm
// bounds the error: an eigenvalue too small to be lifted leaves at most itself.
// Above the tolerance, eight more lifts and a finish follow, up to kMaxLifts in
// all (2.46^40 = 4e15).  The projections are (Y + Q) / 2 and (Y - Q) / 2, both
// positive semidefinite for any X with eigenvalues in [-1, 1] of the right sign.
// Products are symmetric: upper tiles only, mirrored when they are stored.
#include <cfloat>

#include <mutex>
#include <vector>

#include "kernels.cuh"

namespace v2g {

namespace {

constexpr int kFinish = 6;
constexpr int kFirstLifts = 10, kMoreLifts = 8, kMaxLifts = 40;
// a X - b X^3 of the lift (a = 1.5 sqrt(3 c), b = a c for c = 0.9) and of the
// finish steps (c = 1 / (1 + l + l^2) for the lower end l, from 0.246 on)
__constant__ double kLift[2] = {2.4647515087732476, 2.2182763578959230};
__constant__ double kFinishAB[kFinish][2] = {
    {2.2729742729451536, 1.7397217278205195}, {1.9270875094504036, 1.0602310935423533},
    {1.6056189197322020, 0.6132303744871545}, {1.5057267368702252, 0.5057486283709065},
    {1.5000164187752736, 0.5000164189549918}, {1.5, 0.5}};

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

__device__ double cta_total(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += red[i];
    return s;
}

// ---- blocks of dimension up to 64: one CTA, everything in shared memory ----
//
// Bound: the FP64 tensor instructions of the products (a block of 50 padded to
// 56: 392 of 256 FMAs each, 1,568 cycles at the SM's 64 FMAs per cycle) and a
// synchronisation after each.  The warps take 8 x 8 tiles because that splits a
// block's few tiles evenly over 16 warps and pads least.  A cold projection of
// five orbitals (blocks up to 50) takes 65 us on a B200 with its A^T y, where
// the cyclic Jacobi eigensolver took 775 (49 rounds a sweep, two
// synchronisations a round); inside a solve, the projection of n = 5 0.29 ->
// 0.08 ms per outer iteration, although Jacobi started from its previous
// eigenvectors there.  Error against 64-bit eigh 1.8e-15 (Jacobi 2.9e-15).

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallTiles = 3;  // 8 x 8 tiles per warp: 36 upper tiles at n = 64

// One warp's upper tiles of C = P Q (symmetric, commuting operands with zero
// padding), as accumulators: tile u covers rows 8 ti[u].., columns 8 tj[u]...
template <int NU>
__device__ __forceinline__ void small_tiles(const double* P, const double* Q, int n8, int ld, const int (&ti)[kSmallTiles],
                                            const int (&tj)[kSmallTiles], double (&acc)[kSmallTiles][2]) {
    const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    const double *a[NU], *b[NU];
#pragma unroll
    for (int u = 0; u < NU; u++) {
        a[u] = P + (8 * ti[u] + r) * ld + c;
        b[u] = Q + (8 * tj[u] + r) * ld + c;
        acc[u][0] = acc[u][1] = 0.0;
    }
#pragma unroll 2
    for (int k = 0; k < n8; k += 8) {
        double av[NU][2], bv[NU][2];
#pragma unroll
        for (int u = 0; u < NU; u++) {
            av[u][0] = a[u][k];
            bv[u][0] = b[u][k];
            av[u][1] = a[u][k + 4];
            bv[u][1] = b[u][k + 4];
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int u = 0; u < NU; u++) dmma(acc[u][0], acc[u][1], av[u][h], bv[u][h]);
    }
}

__device__ __forceinline__ void small_product(const double* P, const double* Q, int n8, int ld, int nu,
                                              const int (&ti)[kSmallTiles], const int (&tj)[kSmallTiles],
                                              double (&acc)[kSmallTiles][2]) {
    if (nu == 1)
        small_tiles<1>(P, Q, n8, ld, ti, tj, acc);
    else if (nu == 2)
        small_tiles<2>(P, Q, n8, ld, ti, tj, acc);
    else if (nu == 3)
        small_tiles<3>(P, Q, n8, ld, ti, tj, acc);
}

// f(row, col, u, h) for the elements of the warp's tiles that are on or above
// the diagonal of the matrix
template <class F>
__device__ __forceinline__ void small_each(int nu, const int (&ti)[kSmallTiles], const int (&tj)[kSmallTiles], F&& f) {
    const int lane = threadIdx.x & 31, r = lane >> 2, c = 2 * (lane & 3);
#pragma unroll
    for (int u = 0; u < kSmallTiles; u++)
        if (u < nu) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = 8 * ti[u] + r, col = 8 * tj[u] + c + h;
                if (row <= col) f(row, col, u, h);
            }
        }
}

// hint (optional, one word per task): lifts that sufficed last time in the low
// byte, calls since the last trial of fewer above it.
__global__ void __launch_bounds__(kSmallThreads, 1)
    small_sign_kernel(const BlockTask* __restrict__ tasks, int B, const double* __restrict__ aty,
                      const double* __restrict__ c, double* x, double* z, const double* __restrict__ mu,
                      const int* __restrict__ mask, int* __restrict__ hint) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[kSmallWarps];
    const BlockTask t = tasks[blockIdx.x];
    const int b = t.inst;
    if (mask && !mask[b]) return;
    const int N = t.n, nt = (N + 7) / 8, n8 = 8 * nt, ld = n8 + 4;  // ld mod 16 = 4 or 12: conflict-free fragments
    double *S = sm, *X = S + n8 * ld, *X2 = X + n8 * ld, *A = X2 + n8 * ld;
    const double m = mu[b];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int ti[kSmallTiles], tj[kSmallTiles], nu = 0;
#pragma unroll
    for (int u = 0; u < kSmallTiles; u++) {
        int k = warp + u * kSmallWarps, i = 0;
        ti[u] = tj[u] = 0;
        if (k < nt * (nt + 1) / 2) {
            while (k >= nt - i) k -= nt - i++;
            ti[u] = i;
            tj[u] = i + k;
            nu = u + 1;
        }
    }
    // U = sym(A^T y - c + mu x), zero padded
    for (int i = threadIdx.x; i < n8 * n8; i += kSmallThreads) {
        const int p = i / n8, q = i % n8;
        double v = 0.0;
        if (p < N && q < N) {
            const int64_t e1 = (t.xoff + (int64_t)p * N + q) * B + b;
            const int64_t e2 = (t.xoff + (int64_t)q * N + p) * B + b;
            v = 0.5 * (((aty[e1] - c[e1]) + m * x[e1]) + ((aty[e2] - c[e2]) + m * x[e2]));
        }
        S[p * ld + q] = v;
    }
    __syncthreads();
    // the smaller of the Frobenius and the row-sum norm, rounded up to a power
    // of two: scaling by it is exact
    double f = 0.0, rmax = 0.0;
    for (int p = warp; p < N; p += kSmallWarps) {
        double rs = 0.0;
        for (int q = lane; q < N; q += 32) {
            const double v = S[p * ld + q];
            rs += fabs(v);
            f += v * v;
        }
        for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
        if (rs > rmax || rs != rs) rmax = rs;  // keeps a NaN
    }
    f = cta_total(f, red);
    __syncthreads();
    if (lane == 0) red[warp] = rmax;
    __syncthreads();
    for (int i = 0; i < kSmallWarps; i++)
        if (red[i] > rmax || red[i] != red[i]) rmax = red[i];
    double nrm = rmax;
    if (f > 1e-280 && f < 1e280) nrm = fmin(nrm, sqrt(f));
    const auto store = [&](int p, int q, double xv, double zv) {
        const int64_t e = (t.xoff + (int64_t)p * N + q) * B + b;
        x[e] = xv;
        z[e] = zv;
    };
    if (!(nrm > 0.0) || !(nrm <= DBL_MAX)) {
        // a zero block, or one with a non-finite entry
        const double v = nrm == 0.0 ? 0.0 : nan("");
        for (int i = threadIdx.x; i < N * N; i += kSmallThreads) store(i / N, i % N, v, v);
        return;
    }
    const int ex = ilogb(nrm) + 1;
    for (int i = threadIdx.x; i < n8 * n8; i += kSmallThreads) {
        const int o = (i / n8) * ld + i % n8;
        const double v = scalbn(S[o], -ex);
        S[o] = v;
        X[o] = v;
    }
    f = scalbn(sqrt(f), -ex);
    if (!(f > 0.0 && f <= DBL_MAX)) f = 1.0;
    const double tol = 1e-15 * sqrt((double)N) * f;
    __syncthreads();
    double acc[kSmallTiles][2];
    // X <- a X - b X^3
    const auto step = [&](double ca, double cb) {
        small_product(X, X, n8, ld, nu, ti, tj, acc);
        small_each(nu, ti, tj, [&](int p, int q, int u, int h) { A[p * ld + q] = A[q * ld + p] = acc[u][h]; });
        __syncthreads();
        small_product(X, A, n8, ld, nu, ti, tj, acc);
        small_each(nu, ti, tj, [&](int p, int q, int u, int h) {
            X2[p * ld + q] = X2[q * ld + p] = ca * X[p * ld + q] - cb * acc[u][h];
        });
        __syncthreads();
        double* s = X;
        X = X2;
        X2 = s;
    };
    const int h0 = hint ? hint[blockIdx.x] : 0;
    int more = (h0 & 255) ? (h0 & 255) : kFirstLifts, lifts = 0, rounds = 0;
    while (true) {
        for (int i = 0; i < more; i++) step(kLift[0], kLift[1]);
        for (int i = 0; i < kFinish; i++) step(kFinishAB[i][0], kFinishAB[i][1]);
        lifts += more;
        rounds++;
        // Y = S X, Q = Y X
        small_product(S, X, n8, ld, nu, ti, tj, acc);
        small_each(nu, ti, tj, [&](int p, int q, int u, int h) { X2[p * ld + q] = X2[q * ld + p] = acc[u][h]; });
        __syncthreads();
        small_product(X2, X, n8, ld, nu, ti, tj, acc);
        double d2 = 0.0;
        small_each(nu, ti, tj, [&](int p, int q, int u, int h) {
            const double d = S[p * ld + q] - acc[u][h];
            d2 += p == q ? d * d : 2.0 * d * d;
        });
        d2 = cta_total(d2, red);
        if (d2 <= tol * tol || lifts >= kMaxLifts) break;
        more = kMoreLifts;
    }
    if (hint && threadIdx.x == 0) {
        // a finish lifts as much as four lifts; every eighth call tries two fewer
        int k = lifts + 4 * (rounds - 1), calls = (h0 >> 8) + 1;
        if (k > kMaxLifts) k = kMaxLifts;
        if (rounds > 1) calls = 0;
        if (calls == 8) {
            k = k > 6 ? k - 2 : 4;
            calls = 0;
        }
        hint[blockIdx.x] = k | calls << 8;
    }
    const double sx = scalbn(0.5, ex) / m, sz = scalbn(0.5, ex);
    small_each(nu, ti, tj, [&](int p, int q, int u, int h) {
        if (q < N) {
            const double y = X2[p * ld + q], xv = (y + acc[u][h]) * sx, zv = (y - acc[u][h]) * sz;
            store(p, q, xv, zv);
            store(q, p, xv, zv);
        }
    });
}

constexpr int kSmallSmem = 4 * 64 * 68 * (int)sizeof(double);

void set_sign_attrs() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return;
    static std::mutex mu;
    static std::vector<char> done;
    std::lock_guard<std::mutex> lk(mu);
    if ((size_t)dev < done.size() && done[dev]) return;
    if (cudaFuncSetAttribute(small_sign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) != cudaSuccess)
        return;
    if ((size_t)dev >= done.size()) done.resize(dev + 1, 0);
    done[dev] = 1;
}

}  // namespace

void launch_small_project(const BlockTask* tasks, int ntasks, int max_n, int B, const double* aty, const double* c,
                          double* x, double* z, const double* mu, const int* mask, cudaStream_t s, int* hint) {
    if (ntasks == 0) return;
    set_sign_attrs();
    const int n8 = (max_n + 7) / 8 * 8;
    const int smem = 4 * n8 * (n8 + 4) * (int)sizeof(double);
    small_sign_kernel<<<ntasks, kSmallThreads, smem, s>>>(tasks, B, aty, c, x, z, mu, mask, hint);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

}  // namespace v2g
