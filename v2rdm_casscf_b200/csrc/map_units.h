// How the rows of a constraint map are dealt to buckets and work units, and
// which unit a CTA takes.  Plain arithmetic shared by the table builder, the
// launchers and the kernels (maps.cu), and checked without a GPU: every row has
// to belong to exactly one unit of the form that the kernel was built for.
#pragma once

#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define V2G_HD __host__ __device__
#else
#define V2G_HD
#endif

namespace v2g {

constexpr int kMaxBuckets = 7;
constexpr int kBucketWidths[kMaxBuckets] = {1, 2, 4, 5, 8, 16, 32};
constexpr int kMidRow = 256, kMidMany = 32;
// Maps with fewer rows are bound by latency at small batches: their rows of 17 to
// 32 entries take a warp each too, instead of one thread.  The table is built once
// for every number of instances, and this is the better side at few of them (B200,
// us for A / A^T, warp and thread: n = 6 with T1, one instance 2.4 / 2.9 and 2.3 /
// 3.6; n = 7, four 3.2 / 3.9 and 3.5 / 4.8; n = 12 DG, one 3.3 / 3.7 and 3.3 /
// 5.5), the other one from sixteen on (n = 5, 64 instances 7.6 / 7.0 and 3.6 / 4.4;
// n = 7, 32 8.3 / 9.4 and 6.8 / 5.2; n = 12 DG, 128 81 / 93 and 82 / 88).
constexpr int kLatencyRows = 1 << 18;

// The bucket of a row of len entries in a map of nrows rows; kMaxBuckets: a
// long row.
inline int row_bucket(int64_t nrows, int64_t len) {
    if (nrows < kLatencyRows && len > 16) return kMaxBuckets;
    int w = 0;
    while (w < kMaxBuckets && kBucketWidths[w] < len) w++;
    return w;
}
// Whether a long row takes a warp (a mid row) instead of a CTA; same: the number
// of long rows of this length.
inline bool row_is_mid(int64_t len, int same) { return len <= kMidRow && (same >= kMidMany || len <= 32); }

// Lanes of a row: one instance each at B = 1, two above.
V2G_HD constexpr int lanes_of(int B) { return (B + 1) / 2; }

// CTA size of a map launch for B instances: whole passes of a row's lanes,
// rounded up to warps, and at least B (the per-instance sums end in thread b < B).
inline int map_threads(int B) {
    const int n = lanes_of(B);
    return (std::max(256 / n * n, B) + 31) & ~31;
}

// Rows per thread of the deep form, by bucket width; one in the plain form.
V2G_HD constexpr int ell_depth(int W) { return W == 1 ? 4 : (W == 2 ? 2 : 1); }
V2G_HD constexpr int unit_passes(bool deep, int W) { return deep ? ell_depth(W) : 1; }

// Work units of one map application in one form (plain or deep): first the long
// rows (a CTA each), then the mid rows (a warp each, 32 instances at a time),
// then the row tiles.  Unit u runs on CTA u % gridDim.x.
struct Blocks {
    int start[kMaxBuckets + 1];  // first unit of each bucket's row tiles; the last: the unit count
    int mid;                     // first mid-row unit
    int midchunks;               // instance chunks of 32 per group of mid rows
};

// CTA `block` of G: its first row tile of bucket bi; the bucket's tile count or
// more when it has none there, -1 when it has none from this bucket on.
V2G_HD inline int first_tile(const Blocks& bl, int bi, int block, int G) {
    int t0 = block - bl.start[bi];
    if (t0 < 0) {
        if (G >= bl.start[kMaxBuckets]) return -1;  // one unit per CTA
        t0 = (t0 % G + G) % G;
    }
    return t0;
}

// Row tiles of bucket i for `rpp` rows per pass.
template <class Map>
int64_t bucket_tiles(const Map& M, int i, int64_t rpp, bool deep) {
    const int64_t per = rpp * unit_passes(deep, M.width[i]);
    return (M.nslots[i] + per - 1) / per;
}

// Whether a map asks for the deep form: packed, and more tiles with one row per
// thread than deep_from (as many as are resident at once; below, the kernel is
// one latency chain, and more CTAs spread it wider).
template <class Map>
bool wants_deep(const Map& M, int B, int threads, int deep_from) {
    if (!M.packed) return false;
    const int64_t rpp = threads / lanes_of(B);
    int64_t tot = 0;
    for (int i = 0; i < M.nb; i++) tot += bucket_tiles(M, i, rpp, false);
    return tot > deep_from;
}

// The units of a map in the given form, which has to be the kernel's.
template <class Map>
Blocks map_blocks(const Map& M, int B, int threads, bool deep) {
    Blocks bl{};
    bl.mid = M.nlong - M.nmid;
    bl.midchunks = (B + 31) / 32;
    const int64_t rpp = threads / lanes_of(B);
    const int warps = threads / 32;
    int acc = bl.mid + (M.nmid + warps - 1) / warps * bl.midchunks;
    for (int i = 0; i < M.nb; i++) {
        bl.start[i] = acc;
        acc += (int)bucket_tiles(M, i, rpp, deep);
    }
    for (int i = M.nb; i <= kMaxBuckets; i++) bl.start[i] = acc;
    return bl;
}

// The units of A and A^T for one kernel that applies both (the persistent CG):
// one form for the two maps, deep only where both ask for it.
// The tables have to be both packed or both not, since one kernel reads both (each
// table is packed by its own coefficients).
template <class Map>
bool loop_applies(const Map& A, const Map& AT) {
    return (A.packed != 0) == (AT.packed != 0);
}
struct LoopUnits {
    bool deep;
    Blocks A, AT;
};
template <class Map>
LoopUnits loop_units(const Map& A, const Map& AT, int B, int threads, int deep_from) {
    LoopUnits u;
    u.deep = wants_deep(A, B, threads, deep_from) && wants_deep(AT, B, threads, deep_from);
    u.A = map_blocks(A, B, threads, u.deep);
    u.AT = map_blocks(AT, B, threads, u.deep);
    return u;
}

}  // namespace v2g
