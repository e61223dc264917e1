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
// Above the tolerance, four more lifts and a finish follow, up to kMaxLifts in
// all (2.46^40 = 4e15).  The projections are (Y + Q) / 2 and (Y - Q) / 2, both
// positive semidefinite for any X with eigenvalues in [-1, 1] of the right sign.
// Products are symmetric: upper tiles only, mirrored when they are stored.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <utility>
#include <vector>

#include "kernels.cuh"
#include "wait.cuh"

namespace v2g {

namespace {

constexpr int kFinish = 6;
constexpr int kFirstLifts = 10, kMoreLifts = 4, kMaxLifts = 40;
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

// The hint for the next call, from this call's (0: none yet) and its rounds: the
// lifts to begin with in the low byte, calls (plus 16) until the next trial in
// the second, and whether this count is a trial.  Every eighth call tries one
// lift fewer; a failed trial goes back and waits 24 calls, and where a count
// that was no trial fails (the tolerance or the spectrum moved), four more, the
// next round's lifts.
__device__ __forceinline__ int next_hint(int hint, int rounds) {
    int k = (hint & 255) ? (hint & 255) : kFirstLifts, calls = hint ? ((hint >> 8) & 255) - 16 : 0;
    int trial = hint >> 16;
    if (rounds == 1) {
        trial = 0;
        if (++calls >= 8) {
            trial = k > 2;
            k -= trial;
            calls = 0;
        }
    } else {
        k = trial ? k + 1 : k + 4 * (rounds - 1);
        calls = trial ? -16 : 0;
        trial = 0;
        if (k > kMaxLifts) k = kMaxLifts;
    }
    return k | (calls + 16) << 8 | trial << 16;
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

// WARPS = 16 alone on its SM; 8 beside the team kernel below, whose CTAs come
// to lie on every SM and leave registers for a CTA of 256 threads only (with 512
// the small blocks ran after the large ones: 0.47 instead of 0.38 ms for the
// projection of n = 10).
constexpr int kSmallWarps = 16, kSmallWarpsBeside = 8;
// 8 x 8 tiles per warp: 36 upper tiles at n = 64
__host__ __device__ constexpr int small_tile_count(int warps) { return (36 + warps - 1) / warps; }

// One warp's upper tiles of C = P Q (symmetric, commuting operands with zero
// padding), as accumulators: tile u covers rows 8 ti[u].., columns 8 tj[u]...
template <int NU, int T>
__device__ __forceinline__ void small_tiles(const double* P, const double* Q, int n8, int ld, const int (&ti)[T],
                                            const int (&tj)[T], double (&acc)[T][2]) {
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

template <int T>
__device__ __forceinline__ void small_product(const double* P, const double* Q, int n8, int ld, int nu,
                                              const int (&ti)[T], const int (&tj)[T], double (&acc)[T][2]) {
    switch (nu) {
        case 1: small_tiles<1>(P, Q, n8, ld, ti, tj, acc); break;
        case 2: small_tiles<2>(P, Q, n8, ld, ti, tj, acc); break;
        case 3: small_tiles<3>(P, Q, n8, ld, ti, tj, acc); break;
        case 4:
            if constexpr (T >= 4) small_tiles<4>(P, Q, n8, ld, ti, tj, acc);
            break;
        case 5:
            if constexpr (T >= 5) small_tiles<5>(P, Q, n8, ld, ti, tj, acc);
            break;
    }
}

// f(row, col, u, h) for the elements of the warp's tiles that are on or above
// the diagonal of the matrix
template <int T, class F>
__device__ __forceinline__ void small_each(int nu, const int (&ti)[T], const int (&tj)[T], F&& f) {
    const int lane = threadIdx.x & 31, r = lane >> 2, c = 2 * (lane & 3);
#pragma unroll
    for (int u = 0; u < T; u++)
        if (u < nu) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = 8 * ti[u] + r, col = 8 * tj[u] + c + h;
                if (row <= col) f(row, col, u, h);
            }
        }
}

// hint (optional, one word per task): see next_hint.
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS == kSmallWarps ? 1 : 2)
    small_sign_kernel(const BlockTask* __restrict__ tasks, int B, const double* __restrict__ aty,
                      const double* __restrict__ c, double* x, double* z, const double* __restrict__ mu,
                      const int* __restrict__ mask, int* __restrict__ hint) {
    constexpr int kT = small_tile_count(WARPS), kThreads = 32 * WARPS;
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[WARPS];
    const BlockTask t = tasks[blockIdx.x];
    const int b = t.inst;
    if (mask && !mask[b]) return;
    const int N = t.n, nt = (N + 7) / 8, n8 = 8 * nt, ld = n8 + 4;  // ld mod 16 = 4 or 12: conflict-free fragments
    double *S = sm, *X = S + n8 * ld, *X2 = X + n8 * ld, *A = X2 + n8 * ld;
    const double m = mu[b];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int ti[kT], tj[kT], nu = 0;
#pragma unroll
    for (int u = 0; u < kT; u++) {
        int k = warp + u * WARPS, i = 0;
        ti[u] = tj[u] = 0;
        if (k < nt * (nt + 1) / 2) {
            while (k >= nt - i) k -= nt - i++;
            ti[u] = i;
            tj[u] = i + k;
            nu = u + 1;
        }
    }
    // U = sym(A^T y - c + mu x), zero padded
    for (int i = threadIdx.x; i < n8 * n8; i += kThreads) {
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
    for (int p = warp; p < N; p += WARPS) {
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
    for (int i = 0; i < WARPS; i++)
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
        for (int i = threadIdx.x; i < N * N; i += kThreads) store(i / N, i % N, v, v);
        return;
    }
    const int ex = ilogb(nrm) + 1;
    for (int i = threadIdx.x; i < n8 * n8; i += kThreads) {
        const int o = (i / n8) * ld + i % n8;
        const double v = scalbn(S[o], -ex);
        S[o] = v;
        X[o] = v;
    }
    f = scalbn(sqrt(f), -ex);
    if (!(f > 0.0 && f <= DBL_MAX)) f = 1.0;
    const double tol = 1e-15 * sqrt((double)N) * f;
    __syncthreads();
    double acc[kT][2];
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
    if (hint && threadIdx.x == 0) hint[blockIdx.x] = next_hint(h0, rounds);
    const double sx = scalbn(0.5, ex) / m, sz = scalbn(0.5, ex);
    small_each(nu, ti, tj, [&](int p, int q, int u, int h) {
        if (q < N) {
            const double y = X2[p * ld + q], xv = (y + acc[u][h]) * sx, zv = (y - acc[u][h]) * sz;
            store(p, q, xv, zv);
            store(q, p, xv, zv);
        }
    });
}

// ---- larger blocks: a team of CTAs per block, one cooperative launch ----------
//
// Every block is worked on by a team of CTAs that share its products 32 x 32
// tile by tile and meet at a barrier of their own after each (bounded waits; the
// launch is cooperative, so a team's CTAs are all resident).  Bound: at one
// instance of ten orbitals the latency of a product (first loads 2,000 cycles,
// a tile's FP64 instructions 1,700 to 3,600, the barrier 3,000); with many
// or large blocks the FP64 rate.  The operands are symmetric, so both panels of
// a tile are rows: 32 x 32 chunks through a four-stage cp.async ring (L2 only:
// other CTAs wrote them).  One projection of ten orbitals (blocks of 100 to 200,
// 34 to 60 products) takes 0.3 ms on a B200, of fifteen (225 to 450) 0.9 ms;
// block Jacobi took 8.0 and 22 ms from cold, at twice the error.
constexpr int kTeamThreads = 256;
constexpr int kTile = 32, kChunkLd = kTile + 4, kRing = 4;
constexpr int kChunk = kTile * kChunkLd;  // one operand's chunk in shared memory

// All CTAs of the team have arrived `target / size` times; false when the wait ran out.
__device__ __forceinline__ bool team_wait(unsigned int* bar, unsigned int target, int* err) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int v = 0;
        unsigned long long start = 0;
        for (long n = 0;; n++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if (wait_is_over(n, start, err)) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
            if (n > 64) __nanosleep(32);
        }
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ void cp_async16(double* dst, const double* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The CTA's share of the upper 32 x 32 tiles of C = P Q (n32 x n32, leading
// dimension ld, symmetric commuting operands): f(row, col, value, e) for every
// element on or above the diagonal, with e = E(row, col) loaded before the K
// loop.  Even and odd K steps of four go to accumulators of their own: two
// chains per element keep eight instructions in flight per SM quarter, with one
// the loop ran at half the FP64 rate.
template <class E, class F>
__device__ __forceinline__ void team_product(const double* P, const double* Q, int ld, int n32, int rank, int size,
                                             double* ring, E&& early, F&& f) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
    const int wr = 8 * (warp & 3), wc = 16 * (warp >> 2);  // the warp's 8 x 16 part of a tile
    const int nt = n32 / kTile, nk = nt;
    for (int u = rank; u < nt * (nt + 1) / 2; u += size) {
        int ti = 0, k = u;
        while (k >= nt - ti) k -= nt - ti++;
        const int tj = ti + k;
        const double* pr = P + (int64_t)ti * kTile * ld;
        const double* qr = Q + (int64_t)tj * kTile * ld;
        auto fetch = [&](int kc) {
            if (kc < nk) {
                double* s = ring + (kc % kRing) * 2 * kChunk;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int e = threadIdx.x + h * kTeamThreads, row = e >> 4, col = 2 * (e & 15);
                    cp_async16(s + row * kChunkLd + col, pr + (int64_t)row * ld + kc * kTile + col);
                    cp_async16(s + kChunk + row * kChunkLd + col, qr + (int64_t)row * ld + kc * kTile + col);
                }
            }
            cp_commit();
        };
        const int row = ti * kTile + wr + r, col = tj * kTile + wc + 2 * c;
        __syncthreads();  // the ring is free
        fetch(0);
        fetch(1);
        fetch(2);
        double ev[2][2];
#pragma unroll
        for (int v = 0; v < 2; v++)
#pragma unroll
            for (int h = 0; h < 2; h++) ev[v][h] = early(row, col + 8 * v + h);
        double acc[2][2][2] = {};
        for (int kc = 0; kc < nk; kc++) {
            cp_wait<2>();
            __syncthreads();
            fetch(kc + 3);
            const double* a = ring + (kc % kRing) * 2 * kChunk + (wr + r) * kChunkLd + c;
            const double* b = ring + (kc % kRing) * 2 * kChunk + kChunk + (wc + r) * kChunkLd + c;
#pragma unroll
            for (int kk = 0; kk < kTile; kk += 8)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const double av = a[kk + 4 * h], b0 = b[kk + 4 * h], b1 = b[8 * kChunkLd + kk + 4 * h];
                    dmma(acc[h][0][0], acc[h][0][1], av, b0);
                    dmma(acc[h][1][0], acc[h][1][1], av, b1);
                }
        }
#pragma unroll
        for (int v = 0; v < 2; v++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (row <= col + 8 * v + h) f(row, col + 8 * v + h, acc[0][v][h] + acc[1][v][h], ev[v][h]);
    }
}

struct SignArgs {
    const BlockTask* tasks;
    const SignTeam* teams;  // waves x gridDim.x
    int waves, B;
    const double *aty, *c, *mu, *atol;
    double *x, *z;
    const int* mask;
    double *S, *X, *X2, *A, *part;
    unsigned int* bar;  // per task, 0 at the launch
    int* hint;
    int* err;
};

__global__ void __launch_bounds__(kTeamThreads, 2) team_sign_kernel(const __grid_constant__ SignArgs g) {
    extern __shared__ __align__(16) double ring[];
    __shared__ double red[kTeamThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int wave = 0; wave < g.waves; wave++) {
        const SignTeam tm = g.teams[(size_t)wave * gridDim.x + blockIdx.x];
        if (tm.task < 0) continue;
        const BlockTask t = g.tasks[tm.task];
        const int b = t.inst, B = g.B, N = t.n, ld = t.np, n32 = (N + kTile - 1) / kTile * kTile;
        if (g.mask && !g.mask[b]) continue;
        const double m = g.mu[b];
        double *S = g.S + t.woff, *X = g.X + t.woff, *X2 = g.X2 + t.woff, *A = g.A + t.woff;
        double* part = g.part + tm.base;
        unsigned int target = 0;
        auto sync = [&]() {
            target += tm.size;
            return team_wait(g.bar + tm.task, target, g.err);
        };
        // the team's sum of v (per CTA in every thread), the same in every CTA
        auto team_sum = [&](double v, double& out) {
            if (threadIdx.x == 0) part[tm.rank] = v;
            if (!sync()) return false;
            double s = 0.0;
            for (int k = threadIdx.x; k < tm.size; k += kTeamThreads) s += __ldcg(part + k);
            out = cta_total(s, red);
            return true;
        };
        // S = sym(A^T y - c + mu x), zero padded to n32; Frobenius norm and largest row sum
        double f = 0.0, rmax = 0.0;
        for (int p = tm.rank * (kTeamThreads / 32) + warp; p < n32; p += tm.size * (kTeamThreads / 32)) {
            double rs = 0.0;
            for (int q = lane; q < n32; q += 32) {
                double v = 0.0;
                if (p < N && q < N) {
                    const int64_t e1 = (t.xoff + (int64_t)p * N + q) * B + b;
                    const int64_t e2 = (t.xoff + (int64_t)q * N + p) * B + b;
                    v = 0.5 * (((g.aty[e1] - g.c[e1]) + m * g.x[e1]) + ((g.aty[e2] - g.c[e2]) + m * g.x[e2]));
                }
                S[(int64_t)p * ld + q] = v;
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
        for (int i = 0; i < kTeamThreads / 32; i++)
            if (red[i] > rmax || red[i] != red[i]) rmax = red[i];
        if (threadIdx.x == 0) part[tm.size + tm.rank] = rmax;
        if (!team_sum(f, f)) return;
        for (int k = 0; k < tm.size; k++) {
            const double v = __ldcg(part + tm.size + k);
            if (v > rmax || v != v) rmax = v;
        }
        double nrm = rmax;
        if (f > 1e-280 && f < 1e280) nrm = fmin(nrm, sqrt(f));
        // the rows of this CTA, both triangles of its tiles: where x and z are written
        auto store = [&](int p, int q, double xv, double zv) {
            const int64_t e = (t.xoff + (int64_t)p * N + q) * B + b;
            g.x[e] = xv;
            g.z[e] = zv;
        };
        if (!(nrm > 0.0) || !(nrm <= DBL_MAX)) {
            const double v = nrm == 0.0 ? 0.0 : nan("");
            for (int64_t i = tm.rank * kTeamThreads + threadIdx.x; i < (int64_t)N * N; i += tm.size * kTeamThreads)
                store((int)(i / N), (int)(i % N), v, v);
            continue;
        }
        const int ex = ilogb(nrm) + 1;
        for (int p = tm.rank * (kTeamThreads / 32) + warp; p < n32; p += tm.size * (kTeamThreads / 32))
            for (int q = lane; q < n32; q += 32) {
                const int64_t o = (int64_t)p * ld + q;
                const double v = scalbn(S[o], -ex);  // this thread wrote it
                S[o] = v;
                X[o] = v;
            }
        f = scalbn(sqrt(f), -ex);
        if (!(f > 0.0 && f <= DBL_MAX)) f = 1.0;
        double tol = 1e-15 * sqrt((double)N) * f;
        if (g.atol) tol = fmax(tol, scalbn(g.atol[tm.task], -ex));
        if (!sync()) return;
        auto put = [&](double* M, int p, int q, double v) {
            M[(int64_t)p * ld + q] = v;
            M[(int64_t)q * ld + p] = v;
        };
        const auto none = [](int, int) { return 0.0; };
        // X <- a X - b X^3
        auto step = [&](double ca, double cb) {
            team_product(X, X, ld, n32, tm.rank, tm.size, ring, none,
                         [&](int p, int q, double v, double) { put(A, p, q, v); });
            if (!sync()) return false;
            team_product(
                X, A, ld, n32, tm.rank, tm.size, ring, [&](int p, int q) { return __ldcg(X + (int64_t)p * ld + q); },
                [&](int p, int q, double v, double xv) { put(X2, p, q, ca * xv - cb * v); });
            if (!sync()) return false;
            double* s = X;
            X = X2;
            X2 = s;
            return true;
        };
        const int h0 = __ldcg(g.hint + tm.task);
        int more = (h0 & 255) ? (h0 & 255) : kFirstLifts, lifts = 0, rounds = 0;
        while (true) {
            for (int i = 0; i < more; i++)
                if (!step(kLift[0], kLift[1])) return;
            for (int i = 0; i < kFinish; i++)
                if (!step(kFinishAB[i][0], kFinishAB[i][1])) return;
            lifts += more;
            rounds++;
            // Y = S X (into X2), Q = Y X (into A)
            team_product(S, X, ld, n32, tm.rank, tm.size, ring, none,
                         [&](int p, int q, double v, double) { put(X2, p, q, v); });
            if (!sync()) return;
            double d2 = 0.0;
            team_product(
                X2, X, ld, n32, tm.rank, tm.size, ring, [&](int p, int q) { return __ldcg(S + (int64_t)p * ld + q); },
                [&](int p, int q, double v, double sv) {
                    const double d = sv - v;
                    d2 += p == q ? d * d : 2.0 * d * d;
                    A[(int64_t)p * ld + q] = v;
                });
            if (!team_sum(cta_total(d2, red), d2)) return;
            if (d2 <= tol * tol || lifts >= kMaxLifts) break;
            more = kMoreLifts;
        }
        if (tm.rank == 0 && threadIdx.x == 0) g.hint[tm.task] = next_hint(h0, rounds);
        // every thread takes the tile elements it computed
        const double sx = scalbn(0.5, ex) / m, sz = scalbn(0.5, ex);
        const int nt = n32 / kTile;
        for (int u = tm.rank; u < nt * (nt + 1) / 2; u += tm.size) {
            int ti = 0, k = u;
            while (k >= nt - ti) k -= nt - ti++;
            const int tj = ti + k;
            for (int e = threadIdx.x; e < kTile * kTile; e += kTeamThreads) {
                const int p = ti * kTile + e / kTile, q = tj * kTile + e % kTile;
                if (p > q || q >= N) continue;
                const double y = __ldcg(X2 + (int64_t)p * ld + q), v = __ldcg(A + (int64_t)p * ld + q);
                const double xv = (y + v) * sx, zv = (y - v) * sz;
                store(p, q, xv, zv);
                store(q, p, xv, zv);
            }
        }
    }
}

constexpr int kSmallSmem = 4 * 64 * 68 * (int)sizeof(double);
constexpr int kTeamSmem = kRing * 2 * kChunk * (int)sizeof(double);

void set_sign_attrs() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return;
    static std::mutex mu;
    static std::vector<char> done;
    std::lock_guard<std::mutex> lk(mu);
    if ((size_t)dev < done.size() && done[dev]) return;
    if (cudaFuncSetAttribute(small_sign_kernel<kSmallWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmallSmem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(small_sign_kernel<kSmallWarpsBeside>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallSmem) != cudaSuccess ||
        cudaFuncSetAttribute(team_sign_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTeamSmem) != cudaSuccess)
        return;
    if ((size_t)dev >= done.size()) done.resize(dev + 1, 0);
    done[dev] = 1;
}

}  // namespace

void launch_small_project(const BlockTask* tasks, int ntasks, int max_n, int B, const double* aty, const double* c,
                          double* x, double* z, const double* mu, const int* mask, cudaStream_t s, int* hint, bool beside) {
    if (ntasks == 0) return;
    set_sign_attrs();
    const int n8 = (max_n + 7) / 8 * 8;
    const int smem = 4 * n8 * (n8 + 4) * (int)sizeof(double);
    if (beside)
        small_sign_kernel<kSmallWarpsBeside>
            <<<ntasks, 32 * kSmallWarpsBeside, smem, s>>>(tasks, B, aty, c, x, z, mu, mask, hint);
    else
        small_sign_kernel<kSmallWarps><<<ntasks, 32 * kSmallWarps, smem, s>>>(tasks, B, aty, c, x, z, mu, mask, hint);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

int sign_grid(int device) {
    static std::mutex mu;
    static std::vector<int> grids;
    std::lock_guard<std::mutex> lk(mu);
    if ((size_t)device < grids.size() && grids[device] >= 0) return grids[device];
    if ((size_t)device >= grids.size()) grids.resize(device + 1, -1);
    int sms = 0, coop = 0, occ = 0, g = 0;
    set_sign_attrs();
    // two CTAs per SM, and room for the small blocks' CTAs beside them on 16 SMs
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && coop &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, team_sign_kernel, kTeamThreads, kTeamSmem) ==
            cudaSuccess &&
        occ >= 1)
        g = std::min(occ, 2) * std::max(1, sms - 16);
    cudaGetLastError();
    return grids[device] = g;
}

int sign_schedule(const std::vector<BlockTask>& tasks, int grid, std::vector<SignTeam>& teams, int64_t& parts) {
    const int n = (int)tasks.size();
    std::vector<int> order(n), size(n, 1);
    std::vector<int64_t> tiles(n);
    double total = 0.0;
    for (int i = 0; i < n; i++) {
        const int64_t nt = (tasks[i].n + kTile - 1) / kTile;
        tiles[i] = nt * (nt + 1) / 2;
        total += (double)tiles[i] * tasks[i].n;
        order[i] = i;
    }
    // time of a block's product: rounds of tiles times K
    auto time = [&](int i, int s) { return (tiles[i] + s - 1) / s * tasks[i].n; };
    if (2 * n <= grid) {
        // few blocks, each with CTAs of its own: the slowest gets the CTAs that
        // save it a round, while there are any
        for (int used = n;;) {
            const int i = *std::max_element(order.begin(), order.end(),
                                            [&](int a, int b) { return time(a, size[a]) < time(b, size[b]); });
            const int64_t rounds = (tiles[i] + size[i] - 1) / size[i];
            if (rounds == 1) break;
            const int want = (int)((tiles[i] + rounds - 2) / (rounds - 1));
            if (used + want - size[i] > grid) break;
            used += want - size[i];
            size[i] = want;
        }
    } else {
        // many: CTAs by each block's share of the work, blocks one after the other
        for (int i = 0; i < n; i++)
            size[i] = (int)std::min<int64_t>(
                tiles[i], std::max(1.0, std::floor((double)tiles[i] * tasks[i].n / (total / grid))));
    }
    // Longest first, each on the CTAs that are free first.  A CTA's list follows
    // the order of placement, so the first unfinished block can always go on:
    // no team waits for one that waits for it.
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return time(a, size[a]) > time(b, size[b]); });
    std::vector<std::vector<SignTeam>> list(grid);
    std::vector<std::pair<int64_t, int>> busy(grid);
    for (int k = 0; k < grid; k++) busy[k] = {0, k};
    parts = 0;
    for (int i : order) {
        std::sort(busy.begin(), busy.end());
        const int64_t end = busy[size[i] - 1].first + time(i, size[i]);
        for (int r = 0; r < size[i]; r++) {
            list[busy[r].second].push_back(SignTeam{i, r, size[i], parts});
            busy[r].first = end;
        }
        parts += 2 * size[i];
    }
    size_t waves = 0;
    for (const auto& l : list) waves = std::max(waves, l.size());
    teams.assign(waves * grid, SignTeam{-1, 0, 0, 0});
    for (int k = 0; k < grid; k++)
        for (size_t w = 0; w < list[k].size(); w++) teams[w * grid + k] = list[k][w];
    return (int)waves;
}

cudaError_t launch_team_sign(const BlockTask* tasks, int ntasks, const SignTeam* teams, int waves, int grid, int B,
                             const double* aty, const double* c, double* x, double* z, const double* mu,
                             const int* mask, const double* atol, double* S, double* X, double* X2, double* A,
                             double* part, unsigned int* bar, int* hint, int* err, cudaStream_t s) {
    if (ntasks == 0) return cudaSuccess;
    set_sign_attrs();
    cudaError_t e = cudaMemsetAsync(bar, 0, ntasks * sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    SignArgs g{tasks, teams, waves, B, aty, c, mu, atol, x, z, mask, S, X, X2, A, part, bar, hint, err};
    void* args[] = {&g};
    e = cudaLaunchCooperativeKernel((const void*)team_sign_kernel, dim3(grid), dim3(kTeamThreads), args, kTeamSmem, s);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return e;
}

}  // namespace v2g
