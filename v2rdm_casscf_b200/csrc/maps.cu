// Constraint maps, CG vector kernels and per-instance reductions (FP64).
//
// The maps A and A^T are applied as gathers over bucketed-ELL tables shared
// by all instances of a group (see kernels.cuh for the layouts).  A^T is
// the transpose of A's table, so every primal element sums its contributing
// constraints itself: no atomics, deterministic order, and the two maps are
// exact adjoints.  The algorithmic traffic of an application is
// 8 * (dimx + nconstraints) bytes per instance.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "kernels.cuh"

namespace v2g {

std::atomic<long> g_kernel_launches{0};

namespace {

constexpr int kThreads = 256;

inline int grid_for(int64_t work, int threads = kThreads) {
    int64_t g = (work + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > 148 * 64) g = 148 * 64;
    return (int)g;
}

constexpr int kRedBlocks = 148 * 4;
constexpr int kSpmvBlocks = 148 * 64;
// resident CTAs of the map kernels (64 registers a thread; three CTAs with 80
// registers: 334 us where four took 319, n = 20, 19 instances)
constexpr int kMapCtasPerSm = 4;

// Thread mapping shared by the map and vector kernels that also reduce: the
// rows are cut into passes of T/B rows; pass k goes to block k % G, where
// thread t handles instance t % B of row t / B.  A thread therefore always
// serves the same instance (per-instance partial sums come out in a fixed
// order) and the rows in flight at any moment form one contiguous window,
// which keeps the gathers of neighbouring rows in L2.
struct Chunk {
    int64_t first, stride, nrows;
    int b, rsub, rows_per_pass;
    bool live;
};
__device__ __forceinline__ Chunk chunk_of(int64_t nrows, int B) {
    Chunk c;
    c.rows_per_pass = blockDim.x / B;
    const int lanes = c.rows_per_pass * B;
    c.b = threadIdx.x % B;
    c.rsub = threadIdx.x / B;
    c.live = threadIdx.x < lanes;
    c.first = (int64_t)blockIdx.x * c.rows_per_pass + c.rsub;
    c.stride = (int64_t)gridDim.x * c.rows_per_pass;
    c.nrows = nrows;
    return c;
}

// Per-instance sum over the CTA of v, where thread t holds instance t % B;
// the sum for instance b is returned to thread b < B (0 elsewhere), in a fixed
// order.  When B divides 32 the lanes of one instance sit at stride B in every
// warp: shuffles fold them, then thread b adds the warps' sums; otherwise
// thread b walks its rows.  The CTA synchronises on entry and on exit, so
// the shared scratch can be reused right away.
__device__ __forceinline__ double cta_instance_sum(double v, int B) {
    __shared__ double sh[kThreads];
    double s = 0.0;
    __syncthreads();
    if ((32 % B) == 0) {
        for (int o = 16; o >= B; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane < B) sh[warp * B + lane] = v;
        __syncthreads();
        if ((int)threadIdx.x < B)
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sh[w * B + threadIdx.x];
    } else {
        sh[threadIdx.x] = v;
        __syncthreads();
        if ((int)threadIdx.x < B) {
            const int rows_per_pass = blockDim.x / B;
            for (int k = 0; k < rows_per_pass; k++) s += sh[threadIdx.x + k * B];
        }
    }
    __syncthreads();
    return s;
}

// Per-instance block partial of v, written to partial[slot * B + b] (slot is
// the block's index among the partial sums, not always blockIdx.x).
__device__ __forceinline__ void block_partial(double v, int B, double* __restrict__ partial, int64_t slot) {
    const double s = cta_instance_sum(v, B);
    if ((int)threadIdx.x < B) partial[slot * B + threadIdx.x] = s;
}

// ---- the map kernels ---------------------------------------------------------
//
// Lanes run along the instances of a row: each of its lanes_of(B) lanes serves
// one instance (B = 1) or two, so that a warp's gather of one table entry
// reads B contiguous doubles per row, and the lanes of one row read the same
// table entry (a broadcast).  With one row per lane and a chunk of instances
// per thread, as before, every lane of every 8-byte load touched its own cache
// line, and the L1 serves one line per clock.  What bounds the kernels now is
// the latency of the chain table entry -> gather -> store (at one small
// instance, beside the launch) and, in a batch, that latency against the loads
// in flight.  In the deep form a thread works on several rows at once, a pass
// of blockDim / lanes rows apart, with eight gathers in flight, and loads the
// table entries of its next tile meanwhile.  The sum of a row runs in slot
// order in one thread, whatever the form.  A and A^T one after the other on a
// B200, before and now:
//   n = 20, 19 instances   706 -> 275 us   (1.3 -> 3.4 TB/s of vector bytes)
//   n = 28, 1 instance     243 ->  83 us
//   n = 8 T2, 3 instances   99 ->  37 us
//   n = 10, 1 instance     11.6 -> 9.8 us
constexpr int kWarps = kThreads / 32;

// How instances map to lanes: one lane each (B = 1), or two instances per
// lane: l and l + (B + 1) / 2 for odd B (contiguous 8-byte loads), 2 l and
// 2 l + 1 for even B (16-byte loads).
enum LaneMode { kOne = 0, kOdd = 1, kEven = 2 };
__host__ __device__ constexpr int lanes_of(int B) { return (B + 1) / 2; }
static LaneMode lane_mode(int B) { return B == 1 ? kOne : ((B & 1) ? kOdd : kEven); }

// Work units of one map application: first the long rows (a CTA each), then
// the mid rows (a warp each, 32 instances at a time), then the row tiles.
// Unit u runs on CTA u % gridDim.x.
struct Blocks {
    int start[kMaxBuckets + 1];  // first unit of each bucket's row tiles; the last: the unit count
    int mid;                     // first mid-row unit
    int midchunks;               // instance chunks of 32 per group of mid rows
    int deep;                    // the deep form: ell_depth(width) rows per thread
};

// Rows per thread of the deep form, by bucket width.
__host__ __device__ constexpr int ell_depth(int W) { return W == 1 ? 4 : (W == 2 ? 2 : 1); }

// One thread's place among the tiles of a bucket.
struct Lane {
    int B, b0, b1;   // instances of this lane (b1 >= B: none)
    int rsub, rpp;   // its row within a pass, rows per pass
    bool on0, on1;   // instances present and not masked
};

template <int MODE>
__device__ __forceinline__ Lane lane_of(int B, const int* mask) {
    Lane L;
    const int n = lanes_of(B), l = (int)threadIdx.x % n;
    L.B = B;
    L.rpp = (int)blockDim.x / n;
    L.rsub = (int)threadIdx.x / n;
    L.b0 = MODE == kEven ? 2 * l : l;
    L.b1 = MODE == kEven ? 2 * l + 1 : (MODE == kOdd ? l + n : B);
    L.on0 = !mask || mask[L.b0];
    L.on1 = MODE != kOne && L.b1 < B && (!mask || mask[L.b1]);
    return L;
}

// Predicated loads without a branch around each (the compiler's form of a
// conditional load costs more instructions than the load): p where ok, else
// the default (-1, 0).  COH: through L2 (ld.global.cg), for vectors that other
// CTAs of the same (persistent) launch write, never from a stale L1 line.
template <bool STREAM>
__device__ __forceinline__ int32_t load_word(const int32_t* p, bool ok) {
    int32_t v;
    if (STREAM)
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.s32 %0, -1;\n\t@q ld.global.cs.b32 %0, [%1];\n\t}"
            : "=&r"(v)
            : "l"(p), "r"((int)ok));
    else
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.s32 %0, -1;\n\t@q ld.global.nc.b32 %0, [%1];\n\t}"
            : "=&r"(v)
            : "l"(p), "r"((int)ok));
    return v;
}
template <bool COH>
__device__ __forceinline__ double load_one(const double* p, bool ok) {
    double v;
    if (COH)
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "@q ld.global.cg.f64 %0, [%1];\n\t}"
            : "=&d"(v)
            : "l"(p), "r"((int)ok)
            : "memory");
    else
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "@q ld.global.nc.f64 %0, [%1];\n\t}"
            : "=&d"(v)
            : "l"(p), "r"((int)ok));
    return v;
}
template <bool COH>
__device__ __forceinline__ double2 load_two(const double* p, bool ok) {
    double2 v;
    if (COH)
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "mov.f64 %1, 0d0000000000000000;\n\t@q ld.global.cg.v2.f64 {%0, %1}, [%2];\n\t}"
            : "=&d"(v.x), "=&d"(v.y)
            : "l"(p), "r"((int)ok)
            : "memory");
    else
        asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "mov.f64 %1, 0d0000000000000000;\n\t@q ld.global.nc.v2.f64 {%0, %1}, [%2];\n\t}"
            : "=&d"(v.x), "=&d"(v.y)
            : "l"(p), "r"((int)ok));
    return v;
}

// What happens to the sum s of row r for instance b.  The returned values are
// summed per instance where kSum is set.

// out = A in
struct EpiStore {
    static constexpr bool kSum = false;
    double* out;
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s) const {
        out[(int64_t)r * B + b] = s;
        return 0.0;
    }
};
// out = coef (A in - sub) + add, each part optional
struct EpiAffine {
    static constexpr bool kSum = false;
    const double* sub;
    const double* coef;
    const double* add;
    double* out;
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s) const {
        const int64_t t = (int64_t)r * B + b;
        if (sub) s -= sub[r];
        if (coef) s *= coef[b];
        if (add) s += add[t];
        out[t] = s;
        return 0.0;
    }
};
// out = A in, summing dotv . out
struct EpiDot {
    static constexpr bool kSum = true;
    const double* dotv;
    double* out;
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s) const {
        const int64_t t = (int64_t)r * B + b;
        out[t] = s;
        return (COH ? __ldcg(dotv + t) : dotv[t]) * s;
    }
};

// The tiles t0, t0 + tstep, ... of bucket bi, whose width is 1, 2, 5 (WB) or a
// multiple of four (WB = 4, nbatch batches of slots).  A bucket has fewer than
// 2^32 table entries (the table has fewer than 2^31, and padding at most
// doubles a row), so table offsets are 32-bit.
template <int WB, int MODE, bool DEEP, bool STREAM, bool PK, bool COH, class Epi>
__device__ __forceinline__ void ell_rows(const DevMap& M, int bi, int nbatch, int t0, int tstep, const Lane& L,
                                         const double* __restrict__ in, const Epi& e, const double* sbook,
                                         double (&dot)[2]) {
    constexpr int R = DEEP ? ell_depth(WB) : 1;
    constexpr int32_t kCol = PK ? (1 << kCodeShift) - 1 : -1;
    static_assert(!DEEP || PK, "the deep form reads packed tables");
    const uint32_t ns = (uint32_t)M.nslots[bi];
    const int32_t* rows = M.rows + M.row_off[bi];
    const int32_t* cols = M.cols + M.ent_off[bi];
    const double* vals = PK ? nullptr : M.vals + M.ent_off[bi];
    const char* in0 = reinterpret_cast<const char*>(in + L.b0);
    const int sB = 8 * L.B, second = 8 * (L.b1 - L.b0);  // bytes between columns, between the lane's instances
    const uint32_t rpp = (uint32_t)L.rpp;
    // 64-bit, so that the position past the last tile cannot wrap around
    int64_t i = (int64_t)t0 * L.rpp * R + L.rsub;
    const int64_t step = (int64_t)tstep * L.rpp * R;
    if (i >= ns) return;
    auto load = [&](uint32_t at, uint32_t k0, bool any, int32_t (&w)[WB][R]) {
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int k = 0; k < WB; k++)
                w[k][j] = load_word<STREAM>(cols + (size_t)((k0 + k) * ns + at + j * rpp), any && at + j * rpp < ns);
    };
    auto rowids = [&](uint32_t at, bool any, int32_t (&r)[R]) {
#pragma unroll
        for (int j = 0; j < R; j++) r[j] = load_word<STREAM>(rows + (size_t)(at + j * rpp), any && at + j * rpp < ns);
    };
    int32_t w[WB][R], r[R];
    load((uint32_t)i, 0, true, w);
    rowids((uint32_t)i, true, r);
    while (true) {
        const int64_t next = i + step;
        const bool more = next < ns;
        double a0[R], a1[R];
        int32_t rn[R];
#pragma unroll
        for (int j = 0; j < R; j++) a0[j] = a1[j] = 0.0;
#pragma unroll 1
        for (int kb = 0; kb < (WB == 4 ? nbatch : 1); kb++) {
            double g0[WB][R], g1[WB][R], v[WB][R];
#pragma unroll
            for (int k = 0; k < WB; k++)
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const bool ok = w[k][j] >= 0;
                    const double* q = reinterpret_cast<const double*>(in0 + (int64_t)(w[k][j] & kCol) * sB);
                    if (MODE == kEven) {
                        const double2 t = load_two<COH>(q, ok);
                        g0[k][j] = t.x;
                        g1[k][j] = t.y;
                    } else {
                        g0[k][j] = load_one<COH>(q, ok);
                        if (MODE == kOdd)
                            g1[k][j] = load_one<COH>(
                                reinterpret_cast<const double*>(reinterpret_cast<const char*>(q) + second),
                                ok && L.b1 < L.B);
                    }
                    if (!PK)
                        v[k][j] = load_one<false>(vals + (size_t)((kb * WB + k) * ns + (uint32_t)i + j * rpp), ok);
                }
            int32_t wn[WB][R];
            if (WB == 4 && kb + 1 < nbatch) {
                load((uint32_t)i, (kb + 1) * WB, true, wn);  // the next batch of slots
            } else if (DEEP) {
                load((uint32_t)next, 0, more, wn);  // the next tile's first
                rowids((uint32_t)next, more, rn);
            }
#pragma unroll
            for (int k = 0; k < WB; k++)
#pragma unroll
                for (int j = 0; j < R; j++) {
                    // a padding slot adds 0 times some coefficient of the book
                    const double c = PK ? sbook[(w[k][j] >> kCodeShift) & (kBookSize - 1)] : v[k][j];
                    a0[j] += c * g0[k][j];
                    if (MODE != kOne) a1[j] += c * g1[k][j];
                    if (DEEP || WB == 4) w[k][j] = wn[k][j];
                }
        }
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (r[j] >= 0) {
                if (L.on0) dot[0] += e.template one<COH>(r[j], L.B, L.b0, a0[j]);
                if (MODE != kOne && L.on1) dot[1] += e.template one<COH>(r[j], L.B, L.b1, a1[j]);
            }
            if (DEEP) r[j] = rn[j];
        }
        if (!more) break;
        i = next;
        if (!DEEP) {
            load((uint32_t)i, 0, true, w);
            rowids((uint32_t)i, true, r);
        }
    }
}

// Per-instance sums over the CTA (thread b < B gets instance b's) of a value
// that warp w holds in lane l for instance c0 + l, l < cnt (0 elsewhere).
__device__ __forceinline__ double warps_to_instances(double v, int c0, int cnt) {
    __shared__ double sh[kWarps][32];
    sh[threadIdx.x >> 5][threadIdx.x & 31] = v;
    __syncthreads();
    double t = 0.0;
    const int l = (int)threadIdx.x - c0;
    if (l >= 0 && l < cnt)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w][l];
    __syncthreads();
    return t;
}

// Mid rows (33 to kMidRow entries): a warp per row and 32 instances; with
// fewer than 17 instances the lanes also share the row's entries (lane l sums
// entries l / B, l / B + 32 / B, ...) and fold by shuffles.  A CTA per row
// (the long form) left the 5,792 such rows of A^T at n = 8 with T2 with 80
// entries on 256 threads each (38 us of a 48 us launch at one instance).
template <bool COH, class Epi>
__device__ __forceinline__ double mid_rows(const DevMap& M, int B, const double* __restrict__ in, const Epi& e,
                                           const int* __restrict__ mask, int group, int chunk) {
    const int lane = threadIdx.x & 31;
    const int m = group * (int)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int c0 = chunk * 32, cnt = B - c0 < 32 ? B - c0 : 32;
    const int n = cnt <= 16 ? 32 / cnt : 1;
    const int l = lane / cnt, b = c0 + lane % cnt;
    double s = 0.0, res = 0.0;
    if (m < M.nmid) {
        const int k0 = M.long_ptr[m], k1 = M.long_ptr[m + 1];
        if (l < n) {
#pragma unroll 8
            for (int k = k0 + l; k < k1; k += n) {
                const double* g = in + (int64_t)__ldg(M.long_col + k) * B + b;
                s += __ldg(M.long_val + k) * (COH ? __ldcg(g) : __ldg(g));
            }
        }
        for (int left = n; left > 1;) {
            const int h = (left + 1) / 2;
            const double o = __shfl_down_sync(0xffffffffu, s, cnt * h);
            if (l < left - h) s += o;
            left = h;
        }
        if (lane < cnt && !(mask && !mask[b])) res = e.template one<COH>(M.long_rows[m], B, b, s);
    }
    return res;
}

// Long rows: one CTA per row; thread t sums entries k = t / B, t / B + T / B,
// ... for instance t % B, then a fixed-order reduction per instance.
template <bool COH, class Epi>
__device__ __forceinline__ double long_row(const DevMap& M, int B, const double* __restrict__ in, const Epi& e,
                                           const int* __restrict__ mask, int lr) {
    const int lanes = blockDim.x / B;
    const int b = threadIdx.x % B;
    const int l = threadIdx.x / B;
    const int k0 = M.long_ptr[lr], k1 = M.long_ptr[lr + 1];
    double s = 0.0;
    if (l < lanes) {
#pragma unroll 4
        for (int k = k0 + l; k < k1; k += lanes) {
            const double* g = in + (int64_t)__ldg(M.long_col + k) * B + b;
            s += __ldg(M.long_val + k) * (COH ? __ldcg(g) : __ldg(g));
        }
    }
    const double t = cta_instance_sum(s, B);
    double acc = 0.0;
    if ((int)threadIdx.x < B && !(mask && !mask[threadIdx.x]))
        acc = e.template one<COH>(M.long_rows[lr], B, (int)threadIdx.x, t);
    return acc;
}

// All the units of this CTA: returns to thread b < B the CTA's sum of the
// optional dot for instance b (fixed order; 0 elsewhere).
template <int MODE, bool DEEP, bool STREAM, bool PK, bool COH, class Epi>
__device__ __forceinline__ double ell_cta(const DevMap& M, const Blocks& bl, int B, const double* __restrict__ in,
                                          const Epi& e, const int* mask, const double* sbook) {
    const int G = (int)gridDim.x;
    double sum = 0.0;  // thread b: instance b
    int u = (int)blockIdx.x;
    for (; u < bl.mid; u += G) {
        const double d = long_row<COH>(M, B, in, e, mask, M.nmid + u);
        if (Epi::kSum) sum += d;
    }
    for (; u < bl.start[0]; u += G) {
        const int chunk = (u - bl.mid) % bl.midchunks, c0 = chunk * 32;
        const double d = mid_rows<COH>(M, B, in, e, mask, (u - bl.mid) / bl.midchunks, chunk);
        if (Epi::kSum) sum += warps_to_instances(d, c0, B - c0 < 32 ? B - c0 : 32);
    }
    const Lane L = lane_of<MODE>(B, mask);
    double dot[2] = {0.0, 0.0};
    if (L.rsub < L.rpp && (L.on0 || L.on1)) {
#pragma unroll 1
        for (int bi = 0; bi < M.nb; bi++) {
            // the first unit of this bucket that is this CTA's
            int t0 = ((int)blockIdx.x - bl.start[bi]) % G;
            if (t0 < 0) t0 += G;
            if (t0 >= bl.start[bi + 1] - bl.start[bi]) continue;
            const int W = M.width[bi];
            if (W == 1)
                ell_rows<1, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else if (W == 2)
                ell_rows<2, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else if (W == 5)
                ell_rows<5, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else
                ell_rows<4, MODE, DEEP, STREAM, PK, COH>(M, bi, W / 4, t0, G, L, in, e, sbook, dot);
        }
    }
    if (Epi::kSum) {
        // two instances per lane: fold each half on its own, then to thread b
        const int n = lanes_of(B);
        const double s0 = cta_instance_sum(dot[0], n);
        if (MODE == kOne) {
            sum += s0;
        } else {
            __shared__ double sh[kThreads];
            const double s1 = cta_instance_sum(dot[1], n);
            if ((int)threadIdx.x < n) {
                sh[MODE == kEven ? 2 * threadIdx.x : threadIdx.x] = s0;
                const int b1 = MODE == kEven ? 2 * (int)threadIdx.x + 1 : (int)threadIdx.x + n;
                if (b1 < B) sh[b1] = s1;
            }
            __syncthreads();
            if ((int)threadIdx.x < B) sum += sh[threadIdx.x];
            __syncthreads();
        }
    }
    return sum;
}

template <int MODE, bool DEEP, bool STREAM, bool PK, class Epi>
__global__ void __launch_bounds__(kThreads, kMapCtasPerSm)
    ell_kernel(const __grid_constant__ DevMap M, const __grid_constant__ Blocks bl, int B,
               const double* __restrict__ in, const __grid_constant__ Epi e, const int* __restrict__ mask,
               double* __restrict__ partial) {
    // the coefficient book of a packed table, in shared memory
    __shared__ double sbook[kBookSize];
    if (PK) {
        if (threadIdx.x < kBookSize) sbook[threadIdx.x] = M.book[threadIdx.x];
        __syncthreads();
    }
    const double s = ell_cta<MODE, DEEP, STREAM, PK, false>(M, bl, B, in, e, mask, sbook);
    if (Epi::kSum && (int)threadIdx.x < B) partial[(int64_t)blockIdx.x * B + threadIdx.x] = s;
}

// Stage 1: block g reduces a contiguous chunk of elements for every instance;
// thread t handles instance t % B on element rows t / B, t / B + T/B, ...
__global__ void reduce_stage1(int mode, int64_t n, int B, const double* __restrict__ u, const double* __restrict__ v,
                              const double* __restrict__ w, const double* __restrict__ row,
                              double* __restrict__ partial) {
    const int rows_per_pass = blockDim.x / B;
    const int lanes = rows_per_pass * B;
    const int b = threadIdx.x % B;
    const int rsub = threadIdx.x / B;
    double acc = 0.0;
    if (threadIdx.x < lanes) {
        const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
        const int64_t e0 = blockIdx.x * chunk;
        const int64_t e1 = (e0 + chunk < n) ? e0 + chunk : n;
        for (int64_t e = e0 + rsub; e < e1; e += rows_per_pass) {
            const int64_t i = e * B + b;
            double term;
            switch (mode) {
                case RED_DOT: term = u[i] * v[i]; break;
                case RED_ED: {
                    double d = (u[i] + v[i]) - w[i];
                    term = d * d;
                    break;
                }
                case RED_EP: {
                    double d = u[i] - row[e];
                    term = d * d;
                    break;
                }
                default: term = u[i] * row[e]; break;
            }
            acc += term;
        }
    }
    const double s = cta_instance_sum(acc, B);
    if ((int)threadIdx.x < B) partial[(int64_t)blockIdx.x * B + threadIdx.x] = s;
}

// Stage 2: one block per instance sums its nblk partials with a fixed tree
// (deterministic), instead of one thread walking a long dependent chain.
__global__ void reduce_stage2(int nblk, int B, const double* __restrict__ partial, double* __restrict__ out) {
    __shared__ double sh[kThreads];
    const int b = blockIdx.x;
    double s = 0.0;
    for (int k = threadIdx.x; k < nblk; k += blockDim.x) s += partial[(int64_t)k * B + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[b] = sh[0];
}

// out[e * B + b] = row ? row[e] : 0 for instances with mask[b] set
__global__ void set_rows_kernel(int64_t n, int B, const double* __restrict__ row, double* __restrict__ out,
                                const int* __restrict__ mask) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (mask && !mask[b]) continue;
        out[t] = row ? row[t / B] : 0.0;
    }
}

__global__ void c_minus_z_kernel(int64_t n, int B, const double* __restrict__ c, double* __restrict__ z,
                                 const int* __restrict__ mask) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (mask && !mask[b]) continue;
        z[t] = -z[t] + c[t];
    }
}

__global__ void cg_extrapolate_kernel(int64_t n, int B, double* __restrict__ y, double* __restrict__ yprev,
                                      const int* __restrict__ mode) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int m = mode[(int)(t % B)];
        if (m == 0) continue;
        const double v = y[t];
        if (m == 2) y[t] = v + (v - yprev[t]);
        yprev[t] = v;
    }
}

// ---- Anderson acceleration (kernels.cuh) ----

__global__ void aa_save_kernel(int64_t nx, int B, const double* __restrict__ x, const double* __restrict__ z,
                               double* __restrict__ w, const int* __restrict__ mode) {
    const int64_t half = nx * B, total = 2 * half;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        if (!mode[(int)(t % B)]) continue;
        w[t] = (t < half) ? x[t] : z[t - half];
    }
}

// Rows e of the state are walked with the chunk mapping of the reducing
// kernels, so each thread keeps one instance and its 2 m dot products come
// out in a fixed order.
template <int MAXM>
__global__ void __launch_bounds__(kThreads) aa_update_kernel(
    int64_t nx, int B, int m, const double* __restrict__ x, const double* __restrict__ z,
    const double* __restrict__ w, double* __restrict__ fprev, double* __restrict__ gprev, double* __restrict__ dF,
    double* __restrict__ dG, const int* __restrict__ mode, const int* __restrict__ slot,
    double* __restrict__ partial) {
    const int64_t nrows = 2 * nx, half = nx * B;
    const size_t col = (size_t)nrows * B;
    const Chunk ch = chunk_of(nrows, B);
    // acc[2 j] = dF_slot.dF_j, acc[2 j + 1] = dF_j.f; f.f in ff (one spare
    // entry keeps every unrolled index of the output loop in bounds)
    double acc[2 * MAXM + 1];
#pragma unroll
    for (int k = 0; k < 2 * MAXM + 1; k++) acc[k] = 0.0;
    double ff = 0.0;
    if (ch.live) {
        const int b = ch.b;
        const int md = mode[b];
        const int s = slot[b];
        if (md) {
            for (int64_t e = ch.first; e < ch.nrows; e += ch.stride) {
                const int64_t t = e * B + b;
                const double g = (e < nx) ? x[t] : z[t - half];
                const double f = g - w[t];
                if (md == 2) {
                    const double df = f - fprev[t];
                    dF[(size_t)s * col + t] = df;
                    dG[(size_t)s * col + t] = g - gprev[t];
#pragma unroll
                    for (int j = 0; j < MAXM; j++) {
                        if (j < m) {
                            const double dj = (j == s) ? df : dF[(size_t)j * col + t];
                            acc[2 * j] += df * dj;
                            acc[2 * j + 1] += dj * f;
                        }
                    }
                }
                ff += f * f;
                fprev[t] = f;
                gprev[t] = g;
            }
        }
    }
    // partial[(k * gridDim.x + block) * B + b] for k <= 2 m
#pragma unroll
    for (int k = 0; k < 2 * MAXM + 1; k++) {
        if (k <= 2 * m) {
            const double sum = cta_instance_sum((k == 2 * m) ? ff : acc[k], B);
            if ((int)threadIdx.x < B) partial[((int64_t)k * gridDim.x + blockIdx.x) * B + threadIdx.x] = sum;
        }
    }
}

// out[k * B + b] = sum over blocks of partial[(k * nblk + block) * B + b], one
// CTA per (k, b), fixed tree order
__global__ void reduce_stage2_multi(int nblk, int B, const double* __restrict__ partial, double* __restrict__ out) {
    __shared__ double sh[kThreads];
    const int k = blockIdx.x / B, b = blockIdx.x % B;
    const double* p = partial + (int64_t)k * nblk * B;
    double s = 0.0;
    for (int i = threadIdx.x; i < nblk; i += blockDim.x) s += p[(int64_t)i * B + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

template <int MAXM>
__global__ void aa_mix_kernel(int64_t nx, int B, int m, double* __restrict__ x, double* __restrict__ z,
                              const double* __restrict__ dG, const double* __restrict__ gamma,
                              const int* __restrict__ mix) {
    const int64_t half = nx * B, total = 2 * half;
    const size_t col = (size_t)total;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (!mix[b]) continue;
        double v = (t < half) ? x[t] : z[t - half];
#pragma unroll
        for (int j = 0; j < MAXM; j++) {
            if (j < m) {
                const double gj = gamma[b * m + j];
                if (gj != 0.0) v -= gj * dG[(size_t)j * col + t];
            }
        }
        if (t < half)
            x[t] = v;
        else
            z[t - half] = v;
    }
}

__global__ void cg_init_kernel(int64_t n, int B, const double* __restrict__ rhs, const double* __restrict__ Ap,
                               double* __restrict__ r, double* __restrict__ p, const CgScalars* __restrict__ cs) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (!cs[b].active) continue;
        const double v = rhs[t] - Ap[t];
        r[t] = v;
        p[t] = v;
    }
}

__global__ void cg_set_rr_kernel(int B, CgScalars* cs, const double* rr, int* n_active) {
    int cnt = 0;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        if (cs[b].active) {
            cs[b].rr = rr[b];
            cs[b].rrmin = rr[b];
            cnt++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (threadIdx.x == 0) *n_active = cnt;
}

__global__ void cg_alpha_kernel(int B, CgScalars* cs, const double* pap) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B || !cs[b].active) return;
    cs[b].pap = pap[b];
    if (!(pap[b] > 0.0)) {
        // p has no component outside the null space of A^T (or r = 0): no step
        cs[b].alpha = 0.0;
        cs[b].active = 0;
        cs[b].stalled = 1;
        return;
    }
    cs[b].alpha = cs[b].rr / pap[b];
}

// y += alpha p ; r -= alpha Ap ; partial[., b] of r.r (cg_solver.cc:159-165)
__global__ void cg_update_yr_kernel(int64_t n, int B, double* __restrict__ y, double* __restrict__ r,
                                    const double* __restrict__ p, const double* __restrict__ Ap,
                                    const CgScalars* __restrict__ cs, double* __restrict__ partial) {
    const Chunk ch = chunk_of(n, B);
    double acc = 0.0;
    if (ch.live) {
        const int b = ch.b;
        const bool act = cs[b].active;
        const double a = cs[b].alpha;
        for (int64_t e = ch.first; e < ch.nrows; e += ch.stride) {
            const int64_t t = e * B + b;
            double rv = r[t];
            if (act) {
                y[t] += a * p[t];
                rv += -a * Ap[t];
                r[t] = rv;
            }
            acc += rv * rv;
        }
    }
    block_partial(acc, B, partial, blockIdx.x);
}

// y += alpha p ; r -= alpha Ap with alpha = r.r / p.Ap computed by every
// thread from the instance's scalars (no separate alpha launch; p.Ap <= 0
// takes no step and the beta kernel stops the instance); partial[., b] of
// r.r.  Block 0 clears the active-instance counter that the beta kernel
// fills.
__global__ void cg_step_yr_kernel(int64_t n, int B, double* __restrict__ y, double* __restrict__ r,
                                  const double* __restrict__ p, const double* __restrict__ Ap,
                                  const CgScalars* __restrict__ cs, const double* __restrict__ pap,
                                  double* __restrict__ partial, int* __restrict__ n_active) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_active = 0;
    const Chunk ch = chunk_of(n, B);
    double acc = 0.0;
    if (ch.live) {
        const int b = ch.b;
        const double pp = pap[b];
        const bool act = cs[b].active && pp > 0.0;
        const double a = act ? cs[b].rr / pp : 0.0;
        for (int64_t e = ch.first; e < ch.nrows; e += ch.stride) {
            const int64_t t = e * B + b;
            double rv = r[t];
            if (act) {
                y[t] += a * p[t];
                rv += -a * Ap[t];
                r[t] = rv;
            }
            acc += rv * rv;
        }
    }
    block_partial(acc, B, partial, blockIdx.x);
}

// The scalars of cg_solver.cc:159-177 after a step with p.Ap = pap and the new
// r.r = rn: alpha, the ||r|| < tol test, beta and the iteration count, the
// stops on p.Ap <= 0 and on residual growth (kCgGrowth).
__device__ __forceinline__ void cg_scalar_step(CgScalars& c, double pap, double rn) {
    c.do_p = 0;
    if (!c.active) return;
    c.pap = pap;
    if (!(c.pap > 0.0)) {
        // p has no component outside the null space of A^T (or r = 0): no step
        c.alpha = 0.0;
        c.active = 0;
        c.stalled = 1;
        return;
    }
    c.alpha = c.rr / c.pap;
    c.rrnew = rn;
    if (!(sqrt(rn) < c.tol)) {
        if (rn > kCgGrowth * c.rrmin) {
            // diverging on the null space of A^T: keep the current y (kernels.cuh)
            c.active = 0;
            c.stalled = 1;
        } else {
            c.beta = rn / c.rr;
            c.rr = rn;
            c.rrmin = fmin(c.rrmin, rn);
            c.do_p = 1;
            c.iter += 1;
            if (c.iter >= c.maxiter) c.active = 0;
        }
    } else {
        c.active = 0;
    }
    if (!isfinite(rn)) c.active = 0;
}

// One block per instance: r.r from the step kernel's partials (fixed tree),
// then the scalars of cg_solver.cc:159-177: alpha, the ||r|| < tol test,
// beta and the iteration count, the stops on p.Ap <= 0 and on residual
// growth (kCgGrowth); counts the instances still iterating into n_active.
__global__ void cg_beta_reduce_kernel(int nblk, int B, const double* __restrict__ partial,
                                      const double* __restrict__ pap, CgScalars* cs, int* n_active) {
    __shared__ double sh[kThreads];
    const int b = blockIdx.x;
    double s = 0.0;
    for (int k = threadIdx.x; k < nblk; k += blockDim.x) s += partial[(int64_t)k * B + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    CgScalars c = cs[b];
    cg_scalar_step(c, pap[b], sh[0]);
    cs[b] = c;
    if (c.active) atomicAdd(n_active, 1);
}

// One warp: per instance, test ||r|| < tol (cg_solver.cc:167-171), else beta
// and iteration count; counts the instances still iterating.
__global__ void cg_beta_kernel(int B, CgScalars* cs, const double* rrnew, int* n_active) {
    int cnt = 0;
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
        CgScalars c = cs[b];
        c.do_p = 0;
        if (c.active) {
            const double rn = rrnew[b];
            const double nrm = sqrt(rn);
            c.rrnew = rn;
            if (!(nrm < c.tol)) {
                if (rn > kCgGrowth * c.rrmin) {
                    // diverging on the null space of A^T: keep the current y (kernels.cuh)
                    c.active = 0;
                    c.stalled = 1;
                } else {
                    c.beta = rn / c.rr;
                    c.rr = rn;
                    c.rrmin = fmin(c.rrmin, rn);
                    c.do_p = 1;
                    c.iter += 1;
                    if (c.iter >= c.maxiter) c.active = 0;
                }
            } else {
                c.active = 0;
            }
            if (!isfinite(rn)) c.active = 0;
        }
        cnt += c.active;
        cs[b] = c;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (threadIdx.x == 0) *n_active = cnt;
}

__global__ void cg_update_p_kernel(int64_t n, int B, double* __restrict__ p, const double* __restrict__ r,
                                   const CgScalars* __restrict__ cs) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (!cs[b].do_p) continue;
        p[t] = cs[b].beta * p[t] + r[t];
    }
}

// ---- persistent CG for small groups ------------------------------------------
//
// One cooperative launch runs a whole CG solve (cg_solver.cc:141-177) for a
// group of at most kLoopMaxB instances: per iteration four phases over the
// whole grid (A^T p; A (A^T p) with the per-unit partials of p.Ap; y += alpha
// p and r -= alpha Ap with per-CTA partials of r.r; p = beta p + r),
// separated by grid barriers.  Every CTA sums the partials itself in the same
// fixed order, so every CTA holds the same scalars and takes the same
// decision to continue; no CTA waits for a value only another CTA computes.
// Vectors written inside the launch are read through L2 (ld.global.cg).
// Each barrier wait is bounded: a wait that runs out sets *err and the CTA
// leaves the kernel; the others then run out at their next wait.

constexpr long kGridWaitPolls = 1L << 25;  // about a second of polling (short sleeps)
constexpr int kLoopCtasPerSm = 3;

struct CgLoopArgs {
    DevMap A, AT;
    Blocks blA, blAT;  // unit layouts of the two maps
    int B;
    int64_t nc;
    double *y, *r, *p, *atp, *ap;
    CgScalars* cs;
    double* part_dot;  // grid x B
    double* part_rr;   // grid x B
    unsigned int* bar;
    int* err;
    int* n_active;
    int* iters;
    int cap;
};

// Arrive at barrier number target / gridDim.x of the launch and wait for all
// CTAs; false when the wait ran out.
__device__ __forceinline__ bool grid_wait(unsigned int* bar, unsigned int target, int* err) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        // release: the CTA's writes (ordered before this by the barrier above)
        // become visible to every CTA that acquires the counter
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned int v = 0;
        for (long n = 0;; n++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if (n >= kGridWaitPolls) {
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

// out[b] = sum over k < n of part[k * B + b] for every instance b < B, the
// same fixed order in every CTA (strided per thread, warp shuffles, warps).
__device__ __forceinline__ void loop_reduce(const double* part, int n, int B, double* out) {
    __shared__ double wsum[kThreads / 32][kLoopMaxB];
    double acc[kLoopMaxB];
#pragma unroll
    for (int b = 0; b < kLoopMaxB; b++) acc[b] = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x)
#pragma unroll
        for (int b = 0; b < kLoopMaxB; b++)
            if (b < B) acc[b] += __ldcg(part + (int64_t)k * B + b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int b = 0; b < kLoopMaxB; b++) {
        double v = acc[b];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) wsum[warp][b] = v;
    }
    __syncthreads();
    if ((int)threadIdx.x < B) {
        double t = 0.0;
        for (int w = 0; w < kThreads / 32; w++) t += wsum[w][threadIdx.x];
        out[threadIdx.x] = t;
    }
    __syncthreads();
}

template <int MODE, bool DEEP, bool PK>
__global__ void __launch_bounds__(kThreads, kLoopCtasPerSm) cg_loop_kernel(const __grid_constant__ CgLoopArgs L) {
    __shared__ double bookA[kBookSize], bookAT[kBookSize];
    __shared__ CgScalars sc[kLoopMaxB];
    __shared__ int sact[kLoopMaxB];
    __shared__ double spap[kLoopMaxB], srn[kLoopMaxB];
    __shared__ int s_any;
    const int B = L.B;
    if (threadIdx.x < kBookSize) {
        bookA[threadIdx.x] = L.A.book[threadIdx.x];
        bookAT[threadIdx.x] = L.AT.book[threadIdx.x];
    }
    if ((int)threadIdx.x < B) {
        sc[threadIdx.x] = L.cs[threadIdx.x];
        sact[threadIdx.x] = sc[threadIdx.x].active;
    }
    __syncthreads();
    const unsigned int G = gridDim.x;
    unsigned int target = 0;
    const EpiStore eAT{L.atp};
    const EpiDot eA{L.p, L.ap};
    int it = 0;
    while (true) {
        if (threadIdx.x == 0) {
            int a = 0;
            for (int b = 0; b < B; b++) a |= sact[b];
            s_any = a;
        }
        __syncthreads();
        if (!s_any || it >= L.cap) break;
        // A^T p
        ell_cta<MODE, DEEP, false, PK, true>(L.AT, L.blAT, B, L.p, eAT, sact, bookAT);
        target += G;
        if (!grid_wait(L.bar, target, L.err)) return;
        // Ap = A (A^T p) and the partials of p.Ap
        {
            const double s = ell_cta<MODE, DEEP, false, PK, true>(L.A, L.blA, B, L.atp, eA, sact, bookA);
            if ((int)threadIdx.x < B) L.part_dot[(int64_t)blockIdx.x * B + threadIdx.x] = s;
        }
        target += G;
        if (!grid_wait(L.bar, target, L.err)) return;
        loop_reduce(L.part_dot, (int)G, B, spap);
        // y += alpha p, r -= alpha Ap (cg_solver.cc:159-165), partials of r.r
        {
            const int rpp = kThreads / B, lanes = rpp * B;
            const int b = threadIdx.x % B, rsub = threadIdx.x / B;
            double acc = 0.0;
            if ((int)threadIdx.x < lanes) {
                const double pp = spap[b];
                const bool act = sc[b].active && pp > 0.0;
                const double a = act ? sc[b].rr / pp : 0.0;
                for (int64_t e = (int64_t)blockIdx.x * rpp + rsub; e < L.nc; e += (int64_t)G * rpp) {
                    const int64_t t = e * B + b;
                    double rv = __ldcg(L.r + t);
                    if (act) {
                        L.y[t] = __ldcg(L.y + t) + a * __ldcg(L.p + t);
                        rv += -a * __ldcg(L.ap + t);
                        L.r[t] = rv;
                    }
                    acc += rv * rv;
                }
            }
            block_partial(acc, B, L.part_rr, blockIdx.x);
        }
        target += G;
        if (!grid_wait(L.bar, target, L.err)) return;
        loop_reduce(L.part_rr, (int)G, B, srn);
        if ((int)threadIdx.x < B) {
            cg_scalar_step(sc[threadIdx.x], spap[threadIdx.x], srn[threadIdx.x]);
            sact[threadIdx.x] = sc[threadIdx.x].active;
        }
        __syncthreads();
        // p = beta p + r where the instance continues (cg_solver.cc:173-176)
        for (int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x; t < L.nc * B; t += (int64_t)G * kThreads) {
            const int b = (int)(t % B);
            if (!sc[b].do_p) continue;
            L.p[t] = sc[b].beta * __ldcg(L.p + t) + __ldcg(L.r + t);
        }
        it++;
        target += G;
        if (!grid_wait(L.bar, target, L.err)) return;
    }
    if (blockIdx.x == 0) {
        if ((int)threadIdx.x < B) L.cs[threadIdx.x] = sc[threadIdx.x];
        if (threadIdx.x == 0) {
            int cnt = 0;
            for (int b = 0; b < B; b++) cnt += sact[b];
            *L.n_active = cnt;
            *L.iters = it;
        }
    }
}

}  // namespace

static int spmv_grid(int64_t nrows, int B) {
    // enough blocks to fill the GPU; rows per block >= rows per pass
    const int64_t rows_per_pass = kThreads / B;
    int64_t g = (nrows + rows_per_pass - 1) / rows_per_pass;
    if (g > kSpmvBlocks) g = kSpmvBlocks;
    return (int)(g < 1 ? 1 : g);
}

// Whether table loads and output stores bypass the caches (streaming hints):
// the autotuner's choice, or streamed from eight instances up.
static bool map_streamed(const DevMap& M, int B) {
    if (M.variant >= 0 && M.variant < kMapVariants) return M.variant == 1;
    return B >= 8;
}

// CTA size for B instances: whole passes of a row's lanes, rounded up to
// warps, and at least B (the per-instance sums end in thread b < B).
static int map_threads(int B) {
    const int n = lanes_of(B);
    return std::max(kThreads / n * n, B) + 31 & ~31;
}

// Units of a map (Blocks).  Small maps (every tile resident at once with one
// row per thread) keep one row per thread: there the kernel is one latency
// chain, and more CTAs spread it wider.
static Blocks map_blocks(const DevMap& M, int B, int threads) {
    Blocks bl{};
    const int64_t rpp = threads / lanes_of(B);
    auto tiles = [&](int i, bool deep) {
        const int64_t per = rpp * (deep ? ell_depth(M.width[i]) : 1);
        return (M.nslots[i] + per - 1) / per;
    };
    int64_t tot = 0;
    for (int i = 0; i < M.nb; i++) tot += tiles(i, false);
    bl.deep = M.packed && tot > 148 * kMapCtasPerSm;
    bl.mid = M.nlong - M.nmid;
    bl.midchunks = (B + 31) / 32;
    const int warps = threads / 32;
    int acc = bl.mid + (M.nmid + warps - 1) / warps * bl.midchunks;
    for (int i = 0; i < M.nb; i++) {
        bl.start[i] = acc;
        acc += (int)tiles(i, bl.deep != 0);
    }
    for (int i = M.nb; i <= kMaxBuckets; i++) bl.start[i] = acc;
    return bl;
}

// Returns the partial sums written per instance (one per CTA, where the
// epilogue sums).
template <class Epi>
static int run_map(const DevMap& M, int B, const double* in, const Epi& e, const int* mask, double* partial,
                   cudaStream_t s) {
    const int threads = map_threads(B);
    const Blocks bl = map_blocks(M, B, threads);
    const int units = bl.start[kMaxBuckets];
    if (units == 0) return 0;
    // as many CTAs as fit on the device at once, each with its share of the units
    const int g = std::min(units, 148 * kMapCtasPerSm);
    const bool st = map_streamed(M, B);
    auto go = [&](auto mode) {
        constexpr int MODE = decltype(mode)::value;
        auto k = bl.deep ? (st ? ell_kernel<MODE, true, true, true, Epi> : ell_kernel<MODE, true, false, true, Epi>)
                         : (M.packed ? ell_kernel<MODE, false, false, true, Epi>
                                     : ell_kernel<MODE, false, false, false, Epi>);
        k<<<g, threads, 0, s>>>(M, bl, B, in, e, mask, partial);
    };
    switch (lane_mode(B)) {
        case kOne: go(std::integral_constant<int, kOne>()); break;
        case kOdd: go(std::integral_constant<int, kOdd>()); break;
        default: go(std::integral_constant<int, kEven>()); break;
    }
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return g;
}

void launch_spmv(const DevMap& A, int B, const double* in, double* out, const double* sub, const double* coef,
                 const double* add, const int* mask, cudaStream_t s) {
    if (sub || coef || add)
        run_map(A, B, in, EpiAffine{sub, coef, add, out}, mask, nullptr, s);
    else
        run_map(A, B, in, EpiStore{out}, mask, nullptr, s);
}

int64_t reduce_partial_size(int B) { return (int64_t)kSpmvBlocks * B; }

void launch_spmv_dot(const DevMap& A, int B, const double* in, double* out, const double* dotv, const int* mask,
                     double* partial, double* dot_out, cudaStream_t s) {
    const int g = run_map(A, B, in, EpiDot{dotv, out}, mask, partial, s);
    reduce_stage2<<<B, kThreads, 0, s>>>(g, B, partial, dot_out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_reduce(ReduceMode mode, int64_t n, int B, const double* u, const double* v, const double* w,
                   const double* row, double* partial, double* out, cudaStream_t s) {
    reduce_stage1<<<kRedBlocks, kThreads, 0, s>>>((int)mode, n, B, u, v, w, row, partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    reduce_stage2<<<B, kThreads, 0, s>>>(kRedBlocks, B, partial, out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_set_rows(int64_t n, int B, const double* row, double* out, const int* mask, cudaStream_t s) {
    set_rows_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, row, out, mask);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_aa_save(int64_t nx, int B, const double* x, const double* z, double* w, const int* mode, cudaStream_t s) {
    aa_save_kernel<<<grid_for(2 * nx * B), kThreads, 0, s>>>(nx, B, x, z, w, mode);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

int64_t aa_partial_size(int64_t nx, int B, int m) { return (int64_t)(2 * m + 1) * spmv_grid(2 * nx, B) * B; }

void launch_aa_update(int64_t nx, int B, int m, const double* x, const double* z, const double* w, double* fprev,
                      double* gprev, double* dF, double* dG, const int* mode, const int* slot, double* partial,
                      double* dots, cudaStream_t s) {
    const int g = spmv_grid(2 * nx, B);
    if (m <= 4)
        aa_update_kernel<4><<<g, kThreads, 0, s>>>(nx, B, m, x, z, w, fprev, gprev, dF, dG, mode, slot, partial);
    else if (m <= 8)
        aa_update_kernel<8><<<g, kThreads, 0, s>>>(nx, B, m, x, z, w, fprev, gprev, dF, dG, mode, slot, partial);
    else
        aa_update_kernel<kAndersonMax><<<g, kThreads, 0, s>>>(nx, B, m, x, z, w, fprev, gprev, dF, dG, mode, slot,
                                                               partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    reduce_stage2_multi<<<(2 * m + 1) * B, kThreads, 0, s>>>(g, B, partial, dots);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_aa_mix(int64_t nx, int B, int m, double* x, double* z, const double* dG, const double* gamma,
                   const int* mix, cudaStream_t s) {
    const int g = grid_for(2 * nx * B);
    if (m <= 4)
        aa_mix_kernel<4><<<g, kThreads, 0, s>>>(nx, B, m, x, z, dG, gamma, mix);
    else if (m <= 8)
        aa_mix_kernel<8><<<g, kThreads, 0, s>>>(nx, B, m, x, z, dG, gamma, mix);
    else
        aa_mix_kernel<kAndersonMax><<<g, kThreads, 0, s>>>(nx, B, m, x, z, dG, gamma, mix);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_cg_extrapolate(int64_t n, int B, double* y, double* yprev, const int* mode, cudaStream_t s) {
    cg_extrapolate_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, y, yprev, mode);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_c_minus_z(int64_t n, int B, const double* c, double* z, const int* mask, cudaStream_t s) {
    c_minus_z_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, c, z, mask);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_cg_init(int64_t n, int B, const double* rhs, const double* Ap, double* r, double* p, const CgScalars* cs,
                    cudaStream_t s) {
    cg_init_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, rhs, Ap, r, p, cs);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_set_rr(int B, CgScalars* cs, const double* rr, int* n_active, cudaStream_t s) {
    cg_set_rr_kernel<<<1, 32, 0, s>>>(B, cs, rr, n_active);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_alpha(int B, CgScalars* cs, const double* pap, cudaStream_t s) {
    cg_alpha_kernel<<<(B + 127) / 128, 128, 0, s>>>(B, cs, pap);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_update_yr(int64_t n, int B, double* y, double* r, const double* p, const double* Ap,
                         const CgScalars* cs, double* partial, double* rr_out, cudaStream_t s) {
    const int g = spmv_grid(n, B);
    cg_update_yr_kernel<<<g, kThreads, 0, s>>>(n, B, y, r, p, Ap, cs, partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    reduce_stage2<<<B, kThreads, 0, s>>>(g, B, partial, rr_out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_step(int64_t n, int B, double* y, double* r, const double* p, const double* Ap, CgScalars* cs,
                    const double* pap, double* partial, int* n_active, cudaStream_t s) {
    const int g = spmv_grid(n, B);
    cg_step_yr_kernel<<<g, kThreads, 0, s>>>(n, B, y, r, p, Ap, cs, pap, partial, n_active);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    cg_beta_reduce_kernel<<<B, kThreads, 0, s>>>(g, B, partial, pap, cs, n_active);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_beta(int B, CgScalars* cs, const double* rrnew, int* n_active, cudaStream_t s) {
    cg_beta_kernel<<<1, 32, 0, s>>>(B, cs, rrnew, n_active);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
// Condition of the device-side CG loop (the body of a WHILE node in the
// group's CUDA graph): another iteration while an instance still iterates,
// and never more than `cap` iterations in all.
__global__ void cg_while_kernel(cudaGraphConditionalHandle h, const int* __restrict__ n_active, int* count,
                                int cap) {
    const int c = *count + 1;
    *count = c;
    cudaGraphSetConditional(h, (*n_active > 0 && c < cap) ? 1u : 0u);
}
void launch_cg_while(cudaGraphConditionalHandle h, const int* n_active, int* count, int cap, cudaStream_t s) {
    cg_while_kernel<<<1, 1, 0, s>>>(h, n_active, count, cap);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}
void launch_cg_update_p(int64_t n, int B, double* p, const double* r, const CgScalars* cs, cudaStream_t s) {
    cg_update_p_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, p, r, cs);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

int cg_loop_grid(int device) {
    static std::mutex mu;
    static std::map<int, int> grid;
    std::lock_guard<std::mutex> lk(mu);
    auto it = grid.find(device);
    if (it != grid.end()) return it->second;
    int sms = 0, coop = 0, occ = 0;
    int g = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && coop &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cg_loop_kernel<kOdd, true, true>, kThreads, 0) == cudaSuccess) {
        // three CTAs per SM (the launch bound): the phases are latency-bound
        // gathers that want the warps
        const int per_sm = std::min(kLoopCtasPerSm, occ);
        if (per_sm >= 1) g = sms * per_sm;
    }
    cudaGetLastError();
    grid[device] = g;
    return g;
}

bool cg_loop_fits(int64_t nc, int B) { return B >= 1 && B <= kLoopMaxB && nc * B <= kLoopMaxElems; }

cudaError_t launch_cg_loop(const DevMap& A, const DevMap& AT, int B, int64_t nc, double* y, double* r, double* p,
                           double* atp, double* ap, CgScalars* cs, double* part_dot, double* part_rr,
                           unsigned int* bar, int* err, int* n_active, int* iters, int cap, int grid,
                           cudaStream_t s) {
    CgLoopArgs L;
    L.A = A;
    L.AT = AT;
    L.blA = map_blocks(L.A, B, kThreads);
    L.blAT = map_blocks(L.AT, B, kThreads);
    L.B = B;
    L.nc = nc;
    L.y = y;
    L.r = r;
    L.p = p;
    L.atp = atp;
    L.ap = ap;
    L.cs = cs;
    L.part_dot = part_dot;
    L.part_rr = part_rr;
    L.bar = bar;
    L.err = err;
    L.n_active = n_active;
    L.iters = iters;
    L.cap = cap;
    void* args[] = {&L};
    auto pick = [&](auto mode) -> const void* {
        constexpr int MODE = decltype(mode)::value;
        if (!A.packed || !AT.packed) return (const void*)cg_loop_kernel<MODE, false, false>;
        return L.blA.deep && L.blAT.deep ? (const void*)cg_loop_kernel<MODE, true, true>
                                         : (const void*)cg_loop_kernel<MODE, false, true>;
    };
    const LaneMode lm = lane_mode(B);
    const void* fn = lm == kOne ? pick(std::integral_constant<int, kOne>())
                                : (lm == kOdd ? pick(std::integral_constant<int, kOdd>())
                                              : pick(std::integral_constant<int, kEven>()));
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kThreads), args, 0, s);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return e;
}

}  // namespace v2g
