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
#include "wait.cuh"

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
// resident CTAs of the map kernels: 64 registers a thread.  Measured with the bare
// store alone (three CTAs with 80 registers: 334 us where four took 319, n = 20,
// 19 instances); the CG's epilogues with two instances per lane spill 200 to 560
// bytes a thread at 64 registers and were not measured with more.
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
    __shared__ double sh[1024];  // the largest CTA
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
// table entries of its next tile meanwhile.  The sum of a row of a bucket runs in
// slot order in one thread, whatever the form; mid and long rows are summed by
// several threads and folded in a fixed order.  A and A^T one after the other on
// a B200, before and now:
//   n = 20, 19 instances   706 -> 275 us   (1.3 -> 3.4 TB/s of vector bytes)
//   n = 28, 1 instance     243 ->  83 us
//   n = 8 T2, 3 instances   99 ->  37 us
//   n = 10, 1 instance     11.6 -> 9.8 us
constexpr int kLoopThreads = 512;  // CTA of the persistent CG
constexpr int kWarps = 32;         // of the largest CTA

// How instances map to lanes: one lane each (B = 1), or two instances per
// lane: l and l + (B + 1) / 2 (contiguous 8-byte loads) for odd B, and for even B
// where the input is not on a 16-byte boundary; 2 l and 2 l + 1 (16-byte loads)
// for even B else.
enum LaneMode { kOne = 0, kOdd = 1, kEven = 2 };
static LaneMode lane_mode(int B) { return B == 1 ? kOne : ((B & 1) ? kOdd : kEven); }

// Sum of v over the CTA, to thread 0: one synchronisation.  The scratch is free
// again after the CTA's next one.
__device__ __forceinline__ double cta_sum(double v) {
    __shared__ double sh[kWarps];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) {
        if (threadIdx.x < (blockDim.x >> 5)) s = sh[threadIdx.x];
        for (int o = kWarps / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    }
    return threadIdx.x == 0 ? s : 0.0;
}

// Slots whose gathers a thread issues together in rows of eight and more: all
// of them where latency counts, four in the deep form (registers: the batch of
// eight made A^T at n = 20 with 19 instances 213 us instead of 151).
__host__ __device__ constexpr int wide_batch(bool deep) { return deep ? 4 : 8; }

// One thread's place among the tiles of a bucket.
struct Lane {
    int B, b0, b1;   // instances of this lane (b1 >= B: none)
    int rsub, rpp;   // its row within a pass, rows per pass
    bool on0, on1;   // instances present and not masked
};

template <int MODE>
__device__ __forceinline__ Lane lane_of(int B) {
    Lane L;
    const int n = MODE == kOne ? 1 : lanes_of(B), l = MODE == kOne ? 0 : (int)threadIdx.x % n;
    L.B = MODE == kOne ? 1 : B;
    L.rpp = (int)blockDim.x / n;
    L.rsub = (int)threadIdx.x / n;
    L.b0 = MODE == kEven ? 2 * l : l;
    L.b1 = MODE == kEven ? 2 * l + 1 : (MODE == kOdd ? l + n : B);
    L.on0 = true;
    L.on1 = MODE != kOne && L.b1 < B;
    return L;
}
template <int MODE, class Epi>
__device__ __forceinline__ void lane_flags(Lane& L, const Epi& e) {
    L.on0 = e.on(L.b0);
    L.on1 = MODE != kOne && L.b1 < L.B && e.on(L.b1);
}

// Programmatic dependent launch: the map kernels let the next kernel of the
// stream start at once, and wait for the previous one before they read a vector
// or a mask, or write anything; only the tables are read before.  That hides the
// launch and the first table loads (A then A^T of one n = 10 instance through the
// C ABI on a B200: 12.0 -> 11.3 us, replayed from a graph 7.9 -> 5.9).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Predicated loads without a branch around each (the compiler's form of a
// conditional load costs more instructions than the load): p where ok, else
// the default (-1, 0).  Table loads (load_word, load_val) are read-only loads that
// the compiler may place before pdl_wait; vectors, which the previous kernel of
// the stream may still be writing until then, are read by load_one and load_two,
// ordered after the wait.  COH: through L2 (ld.global.cg), for vectors that other
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
__device__ __forceinline__ double load_val(const double* p, bool ok) {
    double v;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
        "@q ld.global.nc.f64 %0, [%1];\n\t}"
        : "=&d"(v)
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
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "@q ld.global.f64 %0, [%1];\n\t}"
            : "=&d"(v)
            : "l"(p), "r"((int)ok)
            : "memory");
    return v;
}
template <bool COH>
__device__ __forceinline__ double load_one(const double* p) {
    double v;
    if (COH)
        asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    else
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
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
        asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
            "mov.f64 %1, 0d0000000000000000;\n\t@q ld.global.v2.f64 {%0, %1}, [%2];\n\t}"
            : "=&d"(v.x), "=&d"(v.y)
            : "l"(p), "r"((int)ok)
            : "memory");
    return v;
}

// What happens to the sum s of row r for instance b: own() loads what the row
// itself needs (issued beside the gathers where a thread has one row), one()
// finishes it; one()'s values are summed per instance where kSum is set.
struct OwnNone {};

// out = A in, for the instances of mask (null: all)
struct EpiStore {
    static constexpr bool kSum = false;
    double* out;
    const int* mask;
    __device__ __forceinline__ bool on(int b) const { return !mask || mask[b]; }
    using Own = OwnNone;
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t, int, int) const {
        return {};
    }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s, const Own&) const {
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
    const int* mask;
    __device__ __forceinline__ bool on(int b) const { return !mask || mask[b]; }
    using Own = OwnNone;
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t, int, int) const {
        return {};
    }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s, const Own&) const {
        const int64_t t = (int64_t)r * B + b;
        if (sub) s -= sub[r];
        if (coef) s *= coef[b];
        if (add) s += add[t];
        out[t] = s;
        return 0.0;
    }
};

// out = A in - coef brow: the right-hand side A (c - z - tau mu x) + tau mu b
// of the dual step with coef = -tau mu
struct EpiRhs {
    static constexpr bool kSum = false;
    const double* brow;
    const double* coef;
    double* out;
    const int* mask;
    using Own = OwnNone;
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t, int, int) const {
        return {};
    }
    __device__ __forceinline__ bool on(int b) const { return !mask || mask[b]; }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s, const Own&) const {
        out[(int64_t)r * B + b] = s - coef[b] * brow[r];
        return 0.0;
    }
};
// sums |A in - brow|^2, stores nothing
struct EpiResidual {
    static constexpr bool kSum = true;
    const double* brow;
    const int* mask;
    using Own = OwnNone;
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t, int, int) const {
        return {};
    }
    __device__ __forceinline__ bool on(int b) const { return !mask || mask[b]; }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s, const Own&) const {
        const double d = s - brow[r];
        return d * d;
    }
};

// The CG iteration (cg_solver.cc:141-177) in two map applications, every
// vector update in the epilogue of the map that produces its input:
//   q = A^T r + beta q   (= A^T p for the new p = r + beta p), summing q.q = p.A A^T p
//   p = r + beta p, y += alpha p, r -= alpha A q, summing r.r
// The textbook order (A^T p, A (A^T p) with p.Ap, then y and r, then p) has
// four passes with a reduction or a barrier after each and moves 12 vectors of
// constraint length and 2 of primal length per iteration; this one has two
// passes and moves 7 and 3 (B200, us per CG iteration: 19 instances of n = 17
// 716 -> 443, 12 of n = 14 227 -> 164, one of n = 20 161 -> 100).  Elements of r, p, y and q other than r's and q's
// gathers are touched only by the thread that owns the row.
struct EpiCgQ {
    static constexpr bool kSum = true;
    const CgScalars* cs;
    double* q;
    struct Own {
        double q;
    };
    __device__ __forceinline__ bool on(int b) const { return cs[b].active; }
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t r, int B, int b) const {
        const double* p = q + (int64_t)r * B + b;
        // beta = 0 in the first iteration, where q holds an earlier solve's values
        return {cs[b].beta != 0.0 ? (COH ? __ldcg(p) : *p) : 0.0};
    }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t r, int B, int b, double s, const Own& o) const {
        s += cs[b].beta * o.q;
        q[(int64_t)r * B + b] = s;
        return s * s;
    }
};
struct EpiCgR {
    static constexpr bool kSum = true;
    const CgScalars* cs;
    double *y, *r, *p;
    struct Own {
        double y, r, p;
    };
    __device__ __forceinline__ bool on(int b) const { return cs[b].step; }
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t row, int B, int b) const {
        const int64_t t = (int64_t)row * B + b;
        Own o;
        o.y = COH ? __ldcg(y + t) : y[t];
        o.r = COH ? __ldcg(r + t) : r[t];
        o.p = 0.0;
        if (cs[b].beta != 0.0) o.p = COH ? __ldcg(p + t) : p[t];
        return o;
    }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t row, int B, int b, double s, const Own& o) const {
        const int64_t t = (int64_t)row * B + b;
        const double alpha = cs[b].alpha;
        const double pv = o.r + cs[b].beta * o.p;
        p[t] = pv;
        y[t] = o.y + alpha * pv;
        const double rv = o.r - alpha * s;
        r[t] = rv;
        return rv * rv;
    }
};
// r = rhs - A (A^T y), summing r.r
struct EpiCgInit {
    static constexpr bool kSum = true;
    const CgScalars* cs;
    const double* rhs;
    double* r;
    struct Own {
        double rhs;
    };
    __device__ __forceinline__ bool on(int b) const { return cs[b].active; }
    template <bool COH>
    __device__ __forceinline__ Own own(int32_t row, int B, int b) const {
        return {rhs[(int64_t)row * B + b]};
    }
    template <bool COH>
    __device__ __forceinline__ double one(int32_t row, int B, int b, double s, const Own& o) const {
        const double rv = o.rhs - s;
        r[(int64_t)row * B + b] = rv;
        return rv * rv;
    }
};

// The tiles t0, t0 + tstep, ... of bucket bi, whose width is 1, 2, 4, 5 (WB) or
// a multiple of eight (nbatch batches of wide_batch slots).  A bucket has fewer than
// 2^32 table entries (the table has fewer than 2^31, and padding at most
// doubles a row), so table offsets are 32-bit.
template <int WB, int MODE, bool DEEP, bool STREAM, bool PK, bool COH, class Epi>
__device__ __forceinline__ void ell_rows(const DevMap& M, int bi, int nbatch, int t0, int tstep, Lane& L,
                                         const double* in, const Epi& e, const double* sbook,
                                         double (&dot)[2]) {
    constexpr int R = unit_passes(DEEP, WB);
    constexpr bool WIDE = WB == wide_batch(DEEP);  // also the bucket of four in the deep form, with one batch
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
    if (!COH) {
        pdl_wait();
        lane_flags<MODE>(L, e);
    }
    while (true) {
        const int64_t next = i + step;
        const bool more = next < ns;
        double a0[R], a1[R];
        int32_t rn[R];
        typename Epi::Own o0[R], o1[R];
#pragma unroll
        for (int j = 0; j < R; j++) a0[j] = a1[j] = 0.0;
        if (!DEEP) {
            if (L.on0) o0[0] = e.template own<COH>(r[0], L.B, L.b0);
            if (MODE != kOne && L.on1) o1[0] = e.template own<COH>(r[0], L.B, L.b1);
        }
#pragma unroll 1
        for (int kb = 0; kb < (WIDE ? nbatch : 1); kb++) {
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
                        v[k][j] = load_val(vals + (size_t)((kb * WB + k) * ns + (uint32_t)i + j * rpp), ok);
                }
            int32_t wn[WB][R];
            if (WIDE && kb + 1 < nbatch) {
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
                    if (DEEP || WIDE) w[k][j] = wn[k][j];
                }
        }
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (r[j] >= 0) {
                if (DEEP && L.on0) o0[j] = e.template own<COH>(r[j], L.B, L.b0);
                if (DEEP && MODE != kOne && L.on1) o1[j] = e.template own<COH>(r[j], L.B, L.b1);
                if (L.on0) dot[0] += e.template one<COH>(r[j], L.B, L.b0, a0[j], o0[j]);
                if (MODE != kOne && L.on1) dot[1] += e.template one<COH>(r[j], L.B, L.b1, a1[j], o1[j]);
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
__device__ __forceinline__ double mid_rows(const DevMap& M, int B, const double* in, const Epi& e,
                                           int group, int chunk) {
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
                s += __ldg(M.long_val + k) * load_one<COH>(g);
            }
        }
        for (int left = n; left > 1;) {
            const int h = (left + 1) / 2;
            const double o = __shfl_down_sync(0xffffffffu, s, cnt * h);
            if (l < left - h) s += o;
            left = h;
        }
        if (lane < cnt && e.on(b)) {
            const int32_t r = M.long_rows[m];
            res = e.template one<COH>(r, B, b, s, e.template own<COH>(r, B, b));
        }
    }
    return res;
}

// Long rows: one CTA per row; thread t sums entries k = t / B, t / B + T / B,
// ... for instance t % B, then a fixed-order reduction per instance.
template <bool COH, class Epi>
__device__ __forceinline__ double long_row(const DevMap& M, int B, const double* in, const Epi& e,
                                           int lr) {
    const int lanes = blockDim.x / B;
    const int b = threadIdx.x % B;
    const int l = threadIdx.x / B;
    const int k0 = M.long_ptr[lr], k1 = M.long_ptr[lr + 1];
    double s = 0.0;
    if (l < lanes) {
#pragma unroll 4
        for (int k = k0 + l; k < k1; k += lanes) {
            const double* g = in + (int64_t)__ldg(M.long_col + k) * B + b;
            s += __ldg(M.long_val + k) * load_one<COH>(g);
        }
    }
    const double t = cta_instance_sum(s, B);
    double acc = 0.0;
    if ((int)threadIdx.x < B && e.on(threadIdx.x)) {
        const int32_t r = M.long_rows[lr];
        acc = e.template one<COH>(r, B, (int)threadIdx.x, t, e.template own<COH>(r, B, (int)threadIdx.x));
    }
    return acc;
}

// All the units of this CTA: returns to thread b < B the CTA's sum of the
// optional dot for instance b (fixed order; 0 elsewhere).
template <int MODE, bool DEEP, bool STREAM, bool PK, bool COH, class Epi>
__device__ __forceinline__ double ell_cta(const DevMap& M, const Blocks& bl, int B, const double* in,
                                          const Epi& e, const double* sbook) {
    const int G = (int)gridDim.x;
    double sum = 0.0;  // thread b: instance b
    int u = (int)blockIdx.x;
    if (!COH && u < bl.start[0]) pdl_wait();
    for (; u < bl.mid; u += G) {
        const double d = long_row<COH>(M, B, in, e, M.nmid + u);
        if (Epi::kSum) sum += d;
    }
    for (; u < bl.start[0]; u += G) {
        const int chunk = (u - bl.mid) % bl.midchunks, c0 = chunk * 32;
        const double d = mid_rows<COH>(M, B, in, e, (u - bl.mid) / bl.midchunks, chunk);
        if (Epi::kSum) sum += warps_to_instances(d, c0, B - c0 < 32 ? B - c0 : 32);
    }
    Lane L = lane_of<MODE>(B);
    if (COH) lane_flags<MODE>(L, e);
    double dot[2] = {0.0, 0.0};
    if (L.rsub < L.rpp && (L.on0 || L.on1)) {
#pragma unroll 1
        for (int bi = 0; bi < M.nb; bi++) {
            const int t0 = first_tile(bl, bi, (int)blockIdx.x, G);
            if (t0 < 0) break;
            if (t0 >= bl.start[bi + 1] - bl.start[bi]) continue;
            const int W = M.width[bi];
            if (W == 1)
                ell_rows<1, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else if (W == 2)
                ell_rows<2, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else if (W == 5)
                ell_rows<5, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else if (W == 4)
                ell_rows<4, MODE, DEEP, STREAM, PK, COH>(M, bi, 1, t0, G, L, in, e, sbook, dot);
            else
                ell_rows<wide_batch(DEEP), MODE, DEEP, STREAM, PK, COH>(M, bi, W / wide_batch(DEEP), t0, G, L, in, e,
                                                                        sbook, dot);
        }
    }
    if (Epi::kSum) {
        if (MODE == kOne) {
            sum += cta_sum(dot[0]);
        } else {
            // two instances per lane: fold each half on its own, then to thread b
            const int n = lanes_of(B);
            const double s0 = cta_instance_sum(dot[0], n);
            __shared__ double sh[256];  // one per instance
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
               const double* in, const __grid_constant__ Epi e, double* __restrict__ partial) {
    pdl_trigger();
    // the coefficient book of a packed table, in shared memory
    __shared__ double sbook[kBookSize];
    if (PK) {
        if (threadIdx.x < kBookSize) sbook[threadIdx.x] = M.book[threadIdx.x];
        __syncthreads();
    }
    const double s = ell_cta<MODE, DEEP, STREAM, PK, false>(M, bl, B, in, e, sbook);
    if (Epi::kSum) {
        pdl_wait();  // a thread without rows has not waited yet
        if ((int)threadIdx.x < B) partial[(int64_t)blockIdx.x * B + threadIdx.x] = s;
    }
}

// Stage 1: block g reduces a contiguous chunk of elements of u . v for every
// instance; thread t handles instance t % B on element rows t / B, t / B + T/B, ...
__global__ void reduce_stage1(int64_t n, int B, const double* __restrict__ u, const double* __restrict__ v,
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
        for (int64_t e = e0 + rsub; e < e1; e += rows_per_pass) acc += u[e * B + b] * v[e * B + b];
    }
    const double s = cta_instance_sum(acc, B);
    if ((int)threadIdx.x < B) partial[(int64_t)blockIdx.x * B + threadIdx.x] = s;
}

// The outer iteration's sums over the primal and dual vectors in one pass, with
// the residual map and one final kernel for all four (nine launches before; n = 5
// on a B200: 72 -> 49 us per outer iteration outside CG and projection, with the
// right-hand side in one map instead of two)
// (v2rdm_solver.cc:1826-1852): partial[k * gridDim.x * B + block * B + b] for
// k = 0 |A^T y + z - c|^2, 1 c . x, 2 b . y.
__global__ void __launch_bounds__(kThreads) sums_kernel(int64_t nx, int64_t nc, int B, const double* __restrict__ aty,
                                                        const double* __restrict__ z, const double* __restrict__ c,
                                                        const double* __restrict__ x, const double* __restrict__ y,
                                                        const double* __restrict__ brow, double* __restrict__ partial) {
    double ed = 0.0, cx = 0.0, by = 0.0;
    const Chunk px = chunk_of(nx, B), py = chunk_of(nc, B);
    if (px.live) {
        for (int64_t e = px.first; e < nx; e += px.stride) {
            const int64_t i = e * B + px.b;
            const double cv = c[i], d = (aty[i] + z[i]) - cv;
            ed += d * d;
            cx += cv * x[i];
        }
        for (int64_t e = py.first; e < nc; e += py.stride) by += y[e * B + py.b] * brow[e];
    }
    const double v[3] = {ed, cx, by};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double s = cta_instance_sum(v[k], B);
        if ((int)threadIdx.x < B) partial[((int64_t)k * gridDim.x + blockIdx.x) * B + threadIdx.x] = s;
    }
}

// red[k * B + b] from the partials of sums_kernel (nsums blocks) and of the
// residual map (nres blocks, after them): ed^2, ep^2, c . x, b . y; one CTA each.
__global__ void errors_kernel(int nsums, int nres, int B, const double* __restrict__ partial,
                              double* __restrict__ red) {
    __shared__ double sh[kThreads];
    const int k = blockIdx.x / B, b = blockIdx.x % B;
    const int part = k == 0 ? 0 : (k == 1 ? 3 : k - 1);
    const int n = k == 1 ? nres : nsums;
    const double* p = partial + (int64_t)part * nsums * B;
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += p[(int64_t)i * B + b];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) red[blockIdx.x] = sh[0];
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

// z <- c - z + coef x (coef = -tau mu): the input of the right-hand side's map;
// with w, w <- (x, z) first for the instances with mode[b] != 0 (the state the
// Anderson step starts from)
__global__ void rhs_input_kernel(int64_t n, int B, const double* __restrict__ c, const double* __restrict__ x,
                                 double* __restrict__ z, const double* __restrict__ coef, const int* __restrict__ mask,
                                 double* __restrict__ w, const int* __restrict__ mode) {
    const int64_t total = n * B;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(t % B);
        if (!mask[b]) continue;
        const double xv = x[t], zv = z[t];
        if (w && mode[b]) {
            w[t] = xv;
            w[total + t] = zv;
        }
        z[t] = (c[t] - zv) + coef[b] * xv;
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

// The scalars of cg_solver.cc:141-177.  After q.q: alpha, unless q is zero or
// rounding noise next to r (p then has no component outside the null space of
// A^T; |p| >= |r|, and the smallest nonzero eigenvalue of A A^T is of order
// 0.1, so a ratio below 1e-26 cannot be anything else): no step.
constexpr double kCgNull = 1e-26;
__device__ __forceinline__ void cg_scalar_alpha(CgScalars& c, double qq) {
    c.pap = qq;
    c.step = c.active && qq > kCgNull * c.rr;
    c.alpha = c.step ? c.rr / qq : 0.0;
}
// After r.r = rn: the ||r|| < tol test, beta and the iteration count, the stop
// without a step and the stop on residual growth (kCgGrowth).
__device__ __forceinline__ void cg_scalar_beta(CgScalars& c, double rn) {
    if (!c.active) return;
    if (!c.step) {
        c.active = 0;
        c.stalled = 1;
        return;
    }
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
            c.iter += 1;
            if (c.iter >= c.maxiter) c.active = 0;
        }
    } else {
        c.active = 0;
    }
    if (!isfinite(rn)) c.active = 0;
}
__device__ __forceinline__ void cg_scalar_rr(CgScalars& c, double rr) {
    if (!c.active) return;
    c.rr = rr;
    c.rrmin = rr;
}

// One block per instance: the sum of a map's per-CTA partials (fixed tree),
// then the scalars: 0 the initial r.r, 1 q.q, 2 the new r.r, which also counts
// the instances still iterating into n_active (cleared by 0 and 1).
__global__ void cg_reduce_kernel(int what, int nblk, int B, const double* __restrict__ partial, CgScalars* cs,
                                 int* n_active) {
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
    if (what == 0) {
        cg_scalar_rr(c, sh[0]);
    } else if (what == 1) {
        cg_scalar_alpha(c, sh[0]);
    } else {
        cg_scalar_beta(c, sh[0]);
        if (c.active) atomicAdd(n_active, 1);
    }
    if (what != 2 && b == 0) *n_active = 0;
    cs[b] = c;
}

// ---- persistent CG for small groups ------------------------------------------
//
// One cooperative launch runs a whole CG solve for a group of at most
// kLoopMaxB instances: q = A^T y and r = rhs - A q, then per iteration the two
// passes of EpiCgQ and EpiCgR, each ended by an exchange of the CTAs' sums that
// is also the grid's barrier.  Bound: the
// exchanges and the latency of the gathers (the vectors sit in L2).  Every CTA
// adds the posted sums itself in the same fixed order, so every CTA holds the same scalars and takes the same decision to continue; no CTA
// waits for a value only another CTA computes.  Vectors written inside the
// launch are read through L2 (ld.global.cg).  Each barrier wait is bounded
// (wait.cuh): a wait that runs out sets *err and the CTA leaves the kernel; the
// others see *err in theirs and leave too.

struct CgLoopArgs {
    DevMap A, AT;
    Blocks blA, blAT;  // unit layouts of the two maps
    int B;
    const double* rhs;
    double *y, *r, *p, *q;
    CgScalars* cs;
    unsigned long long* slots;  // three sets of grid x B
    int* err;
    int* n_active;
    int* iters;
    int cap;
};

// Grid barrier and per-instance sum in one: every CTA posts its value of each
// instance (thread b < B holds instance b's) in its slot of the phase's set,
// the CTA's threads wait for all the slots and add them (the same fixed order
// in every CTA), then after(b, sum) runs in thread b.  A post is a release and
// the poll an acquire, so what the CTAs wrote before is visible after.  Three
// sets take turns: once a CTA has seen all posts of phase k, every CTA is done
// with the set of phase k - 1, and the CTA empties its slots there before it
// posts phase k + 1; the set is used again in phase k + 2.  Beside a counter
// barrier and a pass over stored partials this saves a round trip to L2 per
// phase.  The polls are spread over the CTA: a lane that polled 14 slots one
// after the other took 13,000 cycles for it.  false when a wait ran out.
// a slot per 128-byte line: packed side by side, 148 CTAs polling ten lines
// took 11,000 cycles for an exchange, spread out 6,000
constexpr int kSlotStride = 16;
constexpr unsigned long long kSlotEmpty = ~0ull;  // cudaMemset(0xff): a NaN that no arithmetic here returns
template <int MODE, class F>
__device__ __forceinline__ bool grid_exchange(unsigned long long* sets, unsigned int& phase, int B, double v, int* err,
                                              F&& after) {
    const int G = (int)gridDim.x, n = G * B, t = (int)threadIdx.x;
    unsigned long long* S = sets + (size_t)(phase % 3) * n * kSlotStride;
    unsigned long long* prev = sets + (size_t)((phase + 2) % 3) * n * kSlotStride;
    phase++;
    __syncthreads();  // every thread's writes come before the posts
    if (t < B) {
        unsigned long long bits = (unsigned long long)__double_as_longlong(v);
        if (bits == kSlotEmpty) bits = 0x7ff8000000000000ull;  // a NaN all the same
        asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(S + ((size_t)blockIdx.x * B + t) * kSlotStride), "l"(bits) : "memory");
    }
    // thread t: instance t % B of CTAs t / B, t / B + T / B, ...
    const int lanes = (int)blockDim.x / B * B;
    double s = 0.0;
    bool fine = true;
    if (t < lanes) {
        long polls = 0;
        unsigned long long start = 0;
        for (int k = t; k < n && fine; k += lanes) {
            unsigned long long bits;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(bits) : "l"(S + (size_t)k * kSlotStride) : "memory");
                if (bits != kSlotEmpty) break;
                if (wait_is_over(polls++, start, err)) {
                    atomicExch(err, 1);
                    fine = false;
                    break;
                }
                if (polls > 64) __nanosleep(32);
            }
            s += __longlong_as_double((long long)bits);
        }
    }
    const double sum = MODE == kOne ? cta_sum(s) : cta_instance_sum(s, B);
    if (t < B) {
        prev[((size_t)blockIdx.x * B + t) * kSlotStride] = kSlotEmpty;
        after(t, sum);
    }
    return __syncthreads_and(fine) != 0;
}

template <int MODE, bool DEEP, bool PK>
__global__ void __launch_bounds__(kLoopThreads, 1) cg_loop_kernel(const __grid_constant__ CgLoopArgs L) {
    __shared__ double bookA[kBookSize], bookAT[kBookSize];
    __shared__ CgScalars sc[kLoopMaxB];
    const int B = MODE == kOne ? 1 : L.B;
    const int b = (int)threadIdx.x;
    if (threadIdx.x < kBookSize) {
        bookA[threadIdx.x] = L.A.book[threadIdx.x];
        bookAT[threadIdx.x] = L.AT.book[threadIdx.x];
    }
    if (b < B) sc[b] = L.cs[b];
    __syncthreads();
    unsigned int phase = 0;
    struct EpiQ0 : EpiStore {  // q = A^T y where the instance is solved for
        const CgScalars* cs;
        __device__ __forceinline__ bool on(int i) const { return cs[i].active; }
    } e0;
    e0.out = L.q;
    e0.mask = nullptr;
    e0.cs = sc;
    ell_cta<MODE, DEEP, false, PK, true>(L.AT, L.blAT, B, L.y, e0, bookAT);
    if (!grid_exchange<MODE>(L.slots, phase, B, 0.0, L.err, [&](int, double) {})) return;
    double s = ell_cta<MODE, DEEP, false, PK, true>(L.A, L.blA, B, L.q, EpiCgInit{sc, L.rhs, L.r}, bookA);
    if (!grid_exchange<MODE>(L.slots, phase, B, s, L.err, [&](int i, double rr) { cg_scalar_rr(sc[i], rr); })) return;
    int it = 0;
    for (; it < L.cap; it++) {
        int any = 0;
        for (int i = 0; i < B; i++) any |= sc[i].active;
        if (!any) break;
        s = ell_cta<MODE, DEEP, false, PK, true>(L.AT, L.blAT, B, L.r, EpiCgQ{sc, L.q}, bookAT);
        if (!grid_exchange<MODE>(L.slots, phase, B, s, L.err, [&](int i, double qq) { cg_scalar_alpha(sc[i], qq); })) return;
        s = ell_cta<MODE, DEEP, false, PK, true>(L.A, L.blA, B, L.q, EpiCgR{sc, L.y, L.r, L.p}, bookA);
        if (!grid_exchange<MODE>(L.slots, phase, B, s, L.err, [&](int i, double rn) { cg_scalar_beta(sc[i], rn); })) return;
    }
    if (blockIdx.x == 0) {
        if (b < B) L.cs[b] = sc[b];
        if (b == 0) {
            int cnt = 0;
            for (int i = 0; i < B; i++) cnt += sc[i].active;
            *L.n_active = cnt;
            *L.iters = it;
        }
    }
}

// ---- resident CG --------------------------------------------------------------
//
// The persistent CG for groups small enough that every row of A and of A^T has
// its own lanes: the table words and the row's elements of q, y, r and p stay
// in registers for the whole solve, and an iteration's phase is one round of
// gathers (through L2, where q and r are published), the sum over the CTA and
// the exchange.  cg_loop_kernel instead reloads the row's words, its elements
// and its output row each time, three L2 round trips of about 900 cycles in a
// row (the acquire of each exchange drops the L1's lines); its slowest CTA
// took 13,000 cycles for a phase at n = 10.  B200, us per CG iteration in a
// solve, four counter barriers per iteration before and now: n = 4 34 -> 8.6,
// n = 5 26.5 -> 8.9, n = 10 27.6 -> 11.5; a phase is about 2,000 cycles of
// gathers and CTA sum and 3,700 (27 CTAs) to 6,000 (148) of exchange.
constexpr int kResWords = 8;       // table words per lane
constexpr int kResThreads = 1024;  // the largest CTA with one instance (64 registers), 768 with several (85)
constexpr int kResClasses = kMaxBuckets + kLongClasses;
constexpr int kResSmem = 2 * kResWords * kResThreads * (int)sizeof(int32_t);  // the words of both maps

// One map's rows dealt to warps: class c has rows of up to 8 g[c] entries, g
// lanes per row and instance (32 / (g B) rows per warp), from warp first[c].
struct ResPlan {
    int n, warps;
    int first[kResClasses], g[kResClasses], rows[kResClasses];
    int bucket[kResClasses];  // ELL bucket, or -1: long rows from row0
    int row0[kResClasses];
};

struct CgResArgs {
    DevMap A, AT;
    ResPlan pA, pAT;
    int B;
    const double* rhs;
    double *y, *r, *q;
    CgScalars* cs;
    unsigned long long* slots;  // three sets of grid x B
    int* err;
    int* n_active;
    int* iters;
    int cap;
};

// A thread's place in one map: its row and instance; its words are in shared
// memory (in registers they spill, and the exchanges drop the L1's lines,
// spilled ones too: eight reloads from L2 one after the other).
struct ResLane {
    int row, b, g, nw;  // row < 0: no row; nw: words in use (of any lane of the warp)
    bool head;          // the lane that ends up with the row's sum
};

__device__ __forceinline__ ResLane res_load(const DevMap& M, const ResPlan& P, int warp, int B,
                                            int32_t (*words)[kResThreads]) {
    const int lane = threadIdx.x & 31;
    ResLane L{-1, lane % B, 1, 0, false};
    for (int j = 0; j < kResWords; j++) words[j][threadIdx.x] = -1;
    if (warp >= P.warps) return L;
    int c = 0;
    while (c + 1 < P.n && warp >= P.first[c + 1]) c++;
    const int gB = P.g[c] * B, rpw = 32 / gB, local = lane / gB, part = lane % gB / B;
    const int slot = (warp - P.first[c]) * rpw + local;
    const bool ok = local < rpw && slot < P.rows[c];
    const int bi = P.bucket[c], k0 = part * kResWords;
    L.g = P.g[c];
    L.head = ok && part == 0;
    L.nw = kResWords;
    if (bi >= 0) {
        const int W = M.width[bi];
        if (W < kResWords) L.nw = W;
        if (ok) {
            L.row = M.rows[M.row_off[bi] + slot];
            for (int j = 0; j < kResWords && k0 + j < W; j++)
                words[j][threadIdx.x] = M.cols[M.ent_off[bi] + (int64_t)(k0 + j) * M.nslots[bi] + slot];
        }
    } else if (ok) {
        const int m = P.row0[c] + slot;
        const int at = M.res_ptr[m], len = M.res_ptr[m + 1] - at;
        L.row = M.res_row[m];
        for (int j = 0; j < kResWords && k0 + j < len; j++) words[j][threadIdx.x] = M.res_word[at + k0 + j];
    }
    return L;
}

// The row's sum (valid in the head lanes).
__device__ __forceinline__ double res_gather(const double* in, const ResLane& L, int B,
                                             const int32_t (*words)[kResThreads], const double* book) {
    double s = 0.0;
    for (int j0 = 0; j0 < L.nw; j0 += 4) {
        int32_t w[4];
        double g[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = words[j0 + j][threadIdx.x];
#pragma unroll
        for (int j = 0; j < 4; j++)
            g[j] = load_one<true>(in + (int64_t)(w[j] & ((1 << kCodeShift) - 1)) * B + L.b, w[j] >= 0);
#pragma unroll
        for (int j = 0; j < 4; j++) s += book[(w[j] >> kCodeShift) & (kBookSize - 1)] * g[j];
    }
    for (int h = L.g / 2; h > 0; h >>= 1) s += __shfl_down_sync(0xffffffffu, s, h * B);
    return s;
}

template <bool ONE>
__global__ void __launch_bounds__(ONE ? kResThreads : 768, 1) cg_resident_kernel(const __grid_constant__ CgResArgs A) {
    __shared__ double bookA[kBookSize], bookAT[kBookSize];
    __shared__ CgScalars sc[kLoopMaxB];
    __shared__ double sums[kResThreads / 32 * kLoopMaxB];
    const int B = ONE ? 1 : A.B;
    const int t = (int)threadIdx.x;
    if (t < kBookSize) {
        bookA[t] = A.A.book[t];
        bookAT[t] = A.AT.book[t];
    }
    if (t < B) sc[t] = A.cs[t];
    const int warp = (t >> 5) * (int)gridDim.x + (int)blockIdx.x;
    extern __shared__ int32_t res_words[];  // kResWords x kResThreads of each map
    auto wx = reinterpret_cast<int32_t (*)[kResThreads]>(res_words), wc = wx + kResWords;
    // this thread's row of A^T and of A
    const ResLane lx = res_load(A.AT, A.pAT, warp, B, wx), lc = res_load(A.A, A.pA, warp, B, wc);
    const int64_t tx = (int64_t)lx.row * B + lx.b, tc = (int64_t)lc.row * B + lc.b;
    double y = 0.0, rhs = 0.0, r = 0.0, p = 0.0, q = 0.0;
    if (lc.head) {
        y = A.y[tc];
        rhs = A.rhs[tc];
    }
    __syncthreads();
    unsigned int phase = 0;
    // per-instance sum of v over the CTA, to thread b
    auto total = [&](double v) {
        if (ONE) return cta_sum(v);
        // lane l holds instance l % B: fold each warp, then the warps
        const int lane = t & 31;
        for (int left = 32 / B; left > 1;) {
            const int h = (left + 1) / 2;
            const double o = __shfl_down_sync(0xffffffffu, v, B * h);
            if (lane / B < left - h) v += o;
            left = h;
        }
        if (lane < B) sums[(t >> 5) * kLoopMaxB + lane] = v;
        __syncthreads();
        double s = 0.0;
        if (t < B)
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) s += sums[w * kLoopMaxB + t];
        return s;
    };
    auto exchange = [&](double v, auto after) {
        return grid_exchange<ONE ? kOne : kOdd>(A.slots, phase, B, v, A.err, after);
    };
    double s = res_gather(A.y, lx, B, wx, bookAT);  // q = A^T y
    if (lx.head && sc[lx.b].active) A.q[tx] = s;
    if (!exchange(0.0, [&](int, double) {})) return;
    s = res_gather(A.q, lc, B, wc, bookA);  // r = rhs - A q
    double v = 0.0;
    if (lc.head && sc[lc.b].active) {
        r = rhs - s;
        A.r[tc] = r;
        v = r * r;
    }
    if (!exchange(total(v), [&](int i, double rr) { cg_scalar_rr(sc[i], rr); })) return;
    int it = 0;
    for (; it < A.cap; it++) {
        int any = 0;
        for (int i = 0; i < B; i++) any |= sc[i].active;
        if (!any) break;
        s = res_gather(A.r, lx, B, wx, bookAT);
        v = 0.0;
        if (lx.head && sc[lx.b].active) {
            q = s + sc[lx.b].beta * q;
            A.q[tx] = q;
            v = q * q;
        }
        if (!exchange(total(v), [&](int i, double qq) { cg_scalar_alpha(sc[i], qq); })) return;
        s = res_gather(A.q, lc, B, wc, bookA);
        v = 0.0;
        if (lc.head && sc[lc.b].step) {
            const double alpha = sc[lc.b].alpha;
            p = r + sc[lc.b].beta * p;
            y += alpha * p;
            r -= alpha * s;
            A.r[tc] = r;
            v = r * r;
        }
        if (!exchange(total(v), [&](int i, double rn) { cg_scalar_beta(sc[i], rn); })) return;
    }
    if (lc.head) A.y[tc] = y;
    if (blockIdx.x == 0) {
        if (t < B) A.cs[t] = sc[t];
        if (t == 0) {
            int cnt = 0;
            for (int i = 0; i < B; i++) cnt += sc[i].active;
            *A.n_active = cnt;
            *A.iters = it;
        }
    }
}

}  // namespace

// Whether the deep form's table loads and output stores bypass the caches
// (streaming hints): the autotuner's choice, or streamed from eight instances up.
// The plain form has no such variant.
static bool map_streamed(const DevMap& M, int B) {
    if (M.variant >= 0 && M.variant < kMapVariants) return M.variant == 1;
    return B >= 8;
}

// Returns the partial sums written per instance (one per CTA, where the
// epilogue sums).
template <class Epi>
static int run_map(const DevMap& M, int B, const double* in, const Epi& e, double* partial, cudaStream_t s) {
    const int threads = map_threads(B);
    const bool deep = wants_deep(M, B, threads, 148 * kMapCtasPerSm);
    const Blocks bl = map_blocks(M, B, threads, deep);
    const int units = bl.start[kMaxBuckets];
    if (units == 0) return 0;
    // as many CTAs as fit on the device at once, each with its share of the units
    const int g = std::min(units, 148 * kMapCtasPerSm);
    const bool st = map_streamed(M, B);
    const LaneMode mode = lane_mode(B) == kEven && ((uintptr_t)in & 15) != 0 ? kOdd : lane_mode(B);
    auto go = [&](auto mode) {
        constexpr int MODE = decltype(mode)::value;
        auto k = deep ? (st ? ell_kernel<MODE, true, true, true, Epi> : ell_kernel<MODE, true, false, true, Epi>)
                      : (M.packed ? ell_kernel<MODE, false, false, true, Epi>
                                  : ell_kernel<MODE, false, false, false, Epi>);
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(g);
        cfg.blockDim = dim3(threads);
        cfg.stream = s;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k, M, bl, B, in, e, partial);
    };
    switch (mode) {
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
        run_map(A, B, in, EpiAffine{sub, coef, add, out, mask}, nullptr, s);
    else
        run_map(A, B, in, EpiStore{out, mask}, nullptr, s);
}

int64_t reduce_partial_size(int B) { return (int64_t)kSpmvBlocks * B; }

void launch_dot(int64_t n, int B, const double* u, const double* v, double* partial, double* out, cudaStream_t s) {
    reduce_stage1<<<kRedBlocks, kThreads, 0, s>>>(n, B, u, v, partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    reduce_stage2<<<B, kThreads, 0, s>>>(kRedBlocks, B, partial, out);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_rhs(const DevMap& A, int64_t nx, int B, const double* c, const double* x, double* z, const double* brow,
                const double* coef, const int* mask, double* w, const int* mode, double* rhs, cudaStream_t s) {
    rhs_input_kernel<<<grid_for(nx * B), kThreads, 0, s>>>(nx, B, c, x, z, coef, mask, w, mode);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    run_map(A, B, z, EpiRhs{brow, coef, rhs, mask}, nullptr, s);
}

void launch_errors(const DevMap& A, int64_t nx, int64_t nc, int B, const double* aty, const double* x, const double* y,
                   const double* z, const double* c, const double* brow, const int* mask, double* partial, double* red,
                   cudaStream_t s) {
    const int rpp = kThreads / B;
    const int g = (int)std::min<int64_t>((std::max(nx, nc) + rpp - 1) / rpp, kRedBlocks);
    sums_kernel<<<g, kThreads, 0, s>>>(nx, nc, B, aty, z, c, x, y, brow, partial);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    const int nres = run_map(A, B, x, EpiResidual{brow, mask}, partial + (int64_t)3 * g * B, s);
    errors_kernel<<<4 * B, kThreads, 0, s>>>(g, nres, B, partial, red);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_set_rows(int64_t n, int B, const double* row, double* out, const int* mask, cudaStream_t s) {
    set_rows_kernel<<<grid_for(n * B), kThreads, 0, s>>>(n, B, row, out, mask);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

// Two CTAs per SM: the 2 m + 1 sums of a CTA cost two synchronisations each, so a
// thread takes as many rows as that leaves it (m = 10 at one instance of n = 10:
// 54 us with one row per thread).
static int aa_grid(int64_t nx, int B) {
    const int rpp = kThreads / B;
    return (int)std::min<int64_t>((2 * nx + rpp - 1) / rpp, 2 * 148);
}

int64_t aa_partial_size(int64_t nx, int B, int m) { return (int64_t)(2 * m + 1) * aa_grid(nx, B) * B; }

void launch_aa_update(int64_t nx, int B, int m, const double* x, const double* z, const double* w, double* fprev,
                      double* gprev, double* dF, double* dG, const int* mode, const int* slot, double* partial,
                      double* dots, cudaStream_t s) {
    const int g = aa_grid(nx, B);
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
static void cg_reduce(int what, int nblk, int B, const double* partial, CgScalars* cs, int* n_active, cudaStream_t s) {
    cg_reduce_kernel<<<B, kThreads, 0, s>>>(what, nblk, B, partial, cs, n_active);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
}

void launch_cg_start(const DevMap& A, int B, const double* q, const double* rhs, double* r, CgScalars* cs,
                     double* partial, int* n_active, cudaStream_t s) {
    cg_reduce(0, run_map(A, B, q, EpiCgInit{cs, rhs, r}, partial, s), B, partial, cs, n_active, s);
}
void launch_cg_direction(const DevMap& AT, int B, const double* r, double* q, CgScalars* cs, double* partial,
                         int* n_active, cudaStream_t s) {
    cg_reduce(1, run_map(AT, B, r, EpiCgQ{cs, q}, partial, s), B, partial, cs, n_active, s);
}
void launch_cg_step(const DevMap& A, int B, const double* q, double* y, double* r, double* p, CgScalars* cs,
                    double* partial, int* n_active, cudaStream_t s) {
    cg_reduce(2, run_map(A, B, q, EpiCgR{cs, y, r, p}, partial, s), B, partial, cs, n_active, s);
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
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cg_loop_kernel<kOdd, true, true>, kLoopThreads, 0) == cudaSuccess &&
        cudaFuncSetAttribute(cg_resident_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem) ==
            cudaSuccess &&
        cudaFuncSetAttribute(cg_resident_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem) ==
            cudaSuccess) {
        // one CTA per SM: an exchange costs by its CTAs (n = 10, one instance:
        // 29.8 us per iteration with 430 CTAs of 256 threads)
        const int per_sm = std::min(1, occ);
        if (per_sm >= 1) g = sms * per_sm;
    }
    cudaGetLastError();
    grid[device] = g;
    return g;
}

size_t cg_loop_slots(int grid, int B) { return 3 * (size_t)grid * B * kSlotStride; }

bool cg_loop_fits(const DevMap& A, const DevMap& AT, int B) {
    return B >= 1 && B <= kLoopMaxB && A.nrows <= kLoopMaxRows && loop_applies(A, AT);
}

// The rows of M dealt to warps for B instances; false when they do not fit
// (unpacked, or rows longer than 8 entries for each of 32 / B lanes).
static bool res_plan(const DevMap& M, int B, ResPlan& P) {
    if (M.nres < 0) return false;
    P = ResPlan{};
    int64_t at = 0;
    auto add = [&](int g, int64_t rows, int bucket, int row0) {
        if (rows == 0) return true;
        if (g * B > 32 || P.n == kResClasses) return false;
        const int rpw = 32 / (g * B);
        P.first[P.n] = (int)at;
        P.g[P.n] = g;
        P.rows[P.n] = (int)rows;
        P.bucket[P.n] = bucket;
        P.row0[P.n] = row0;
        P.n++;
        at += (rows + rpw - 1) / rpw;
        return at < (1 << 24);
    };
    for (int i = 0; i < M.nb; i++)
        if (!add(std::max(1, M.width[i] / kResWords), M.nslots[i], i, 0)) return false;
    // the long rows, sorted by length
    int row0 = 0;
    for (int c = 0; c < kLongClasses; c++) {
        if (!add(2 << c, M.res_upto[c] - row0, -1, row0)) return false;
        row0 = M.res_upto[c];
    }
    P.warps = (int)at;
    return true;
}

static bool cg_resident(const DevMap& A, const DevMap& AT, int B, int sms, ResPlan& pA, ResPlan& pAT, int& grid,
                        int& threads) {
    if (!res_plan(A, B, pA) || !res_plan(AT, B, pAT)) return false;
    const int warps = std::max(pA.warps, pAT.warps);
    // eight warps per CTA while the device has SMs for them
    grid = std::min(sms, std::max(1, (warps + 7) / 8));
    threads = 32 * ((warps + grid - 1) / grid);
    return threads <= (B == 1 ? kResThreads : 768);
}

cudaError_t launch_cg_loop(const DevMap& A, const DevMap& AT, int B, const double* rhs, double* y, double* r, double* p,
                           double* q, CgScalars* cs, unsigned long long* slots, int* err, int* n_active,
                           int* iters, int cap, int grid, cudaStream_t s) {
    cudaError_t e;
    ResPlan pA, pAT;
    int rgrid = 0, rthreads = 0;
    if (cg_resident(A, AT, B, grid, pA, pAT, rgrid, rthreads)) {
        e = cudaMemsetAsync(slots, 0xff, cg_loop_slots(rgrid, B) * sizeof(*slots), s);
        if (e != cudaSuccess) return e;
        CgResArgs R{A, AT, pA, pAT, B, rhs, y, r, q, cs, slots, err, n_active, iters, cap};
        void* args[] = {&R};
        const void* fn = B == 1 ? (const void*)cg_resident_kernel<true> : (const void*)cg_resident_kernel<false>;
        e = cudaLaunchCooperativeKernel(fn, dim3(rgrid), dim3(rthreads), args, kResSmem, s);
        g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
        return e;
    }
    CgLoopArgs L;
    L.A = A;
    L.AT = AT;
    const LoopUnits units = loop_units(A, AT, B, kLoopThreads, 4 * grid);
    L.blA = units.A;
    L.blAT = units.AT;
    // no more CTAs than the larger map has units: a barrier costs by its CTAs
    grid = std::min(grid, std::max(L.blA.start[kMaxBuckets], L.blAT.start[kMaxBuckets]));
    L.B = B;
    L.rhs = rhs;
    L.y = y;
    L.r = r;
    L.p = p;
    L.q = q;
    L.cs = cs;
    L.slots = slots;
    L.err = err;
    L.n_active = n_active;
    L.iters = iters;
    L.cap = cap;
    e = cudaMemsetAsync(slots, 0xff, cg_loop_slots(grid, B) * sizeof(*slots), s);
    if (e != cudaSuccess) return e;
    void* args[] = {&L};
    auto pick = [&](auto mode) -> const void* {
        constexpr int MODE = decltype(mode)::value;
        if (!A.packed) return (const void*)cg_loop_kernel<MODE, false, false>;
        return units.deep ? (const void*)cg_loop_kernel<MODE, true, true>
                          : (const void*)cg_loop_kernel<MODE, false, true>;
    };
    const LaneMode lm = lane_mode(B);
    const void* fn = lm == kOne ? pick(std::integral_constant<int, kOne>())
                                : (lm == kOdd ? pick(std::integral_constant<int, kOdd>())
                                              : pick(std::integral_constant<int, kEven>()));
    e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kLoopThreads), args, 0, s);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return e;
}

}  // namespace v2g
