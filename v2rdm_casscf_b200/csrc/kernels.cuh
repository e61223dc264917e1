// Device kernels of the boundary-point SDP solver (declarations of the
// host-side launchers).
//
// Vector layout: a group of B instances that share one constraint layout is
// stored instance-interleaved, element e of instance b at [e * B + b].  A
// gather through the shared index tables then reads B contiguous doubles per
// table entry, and the table itself is read once for all B instances.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <vector>

#include "map_units.h"

namespace v2g {

// Number of kernels the launchers below have issued (all threads, all devices).
extern std::atomic<long> g_kernel_launches;

// A sparse map (A or A^T) in bucketed ELL form: rows are grouped by length
// into buckets of fixed width (1, 2, 4, 5, 8, 16, 32 slots, padding marked by
// col = -1; the spin rows of A have five entries), stored slot-major so that a warp reads its table entries
// coalesced and needs no row-pointer lookup; rows longer than 32 entries
// (traces, contractions) are kept as CSR, the first nmid of them (at most
// kMidRow entries, kMidMany or more rows of the same length) reduced by a warp
// each, the others by a whole CTA.
constexpr int kLongClasses = 5;  // rows of up to 16, 32, 64, 128 and 256 entries
constexpr int kCodeShift = 27;                 // packed entry: 27 column bits, 4 code bits
constexpr int kBookSize = 1 << (31 - kCodeShift);  // 16 coefficients at most
struct DevMap {
    int64_t nrows = 0;  // output length
    int nb = 0;
    int width[kMaxBuckets] = {};
    int64_t nslots[kMaxBuckets] = {};
    int64_t row_off[kMaxBuckets] = {};  // into rows
    int64_t ent_off[kMaxBuckets] = {};  // into cols / vals
    const int32_t* rows = nullptr;
    // Entry words.  Packed: column | code << kCodeShift, the coefficient
    // book[code] (the maps have a handful of distinct coefficients: +-1,
    // +-1/2, -1/sqrt 2, a few small integers), 4 bytes per entry instead of
    // 12.  Unpacked (a table whose columns or coefficients do not fit): the
    // column, with vals[] the coefficient.  Padding slots are -1 in both forms.
    const int32_t* cols = nullptr;
    const double* vals = nullptr;
    int packed = 0;
    double book[kBookSize] = {};
    int nlong = 0, nmid = 0;
    const int32_t* long_rows = nullptr;
    const int32_t* long_ptr = nullptr;
    const int32_t* long_col = nullptr;
    const double* long_val = nullptr;
    // the same rows sorted by length with packed entries, for the resident CG
    // (a packed table with no row above 256 entries; else nres = -1), and the
    // end of each length class among them
    int nres = -1;
    int res_upto[kLongClasses] = {};
    const int32_t* res_row = nullptr;
    const int32_t* res_ptr = nullptr;
    const int32_t* res_word = nullptr;
    // kernel variant chosen by the autotuner for one instance count (-1: the
    // built-in rule); see kMapVariants
    int variant = -1;
};
// Map kernel variants: whether the table loads and output stores bypass the
// caches (streaming hints).
constexpr int kMapVariants = 2;  // 0: plain, 1: streamed

// out[r,b] = coef[b] * (sum_k val[k] in[col[k],b] - sub[r]) + add[r,b]
// (each of sub, coef, add optional); instances with mask[b] == 0 are skipped.
void launch_spmv(const DevMap& A, int B, const double* in, double* out, const double* sub, const double* coef,
                 const double* add, const int* mask, cudaStream_t s);

// out[b] = u . v per instance over interleaved vectors of n elements
// (deterministic).  partial holds reduce_partial_size(B) doubles.
void launch_dot(int64_t n, int B, const double* u, const double* v, double* partial, double* out, cudaStream_t s);
int64_t reduce_partial_size(int B);

// The right-hand side of the dual step (v2rdm_solver.cc:1783-1794) for the
// instances of mask: z <- c - z + coef x with coef = -tau mu, rhs = A z - coef b.
// The reference forms A (c - z) and -tau mu (A x - b) apart; one map does both.
// With w (2 nx rows), w <- (x, z) before, where mode[b] != 0.
void launch_rhs(const DevMap& A, int64_t nx, int B, const double* c, const double* x, double* z, const double* brow,
                const double* coef, const int* mask, double* w, const int* mode, double* rhs, cudaStream_t s);

// red[0..B) = |A^T y + z - c|^2, red[B..) = |A x - b|^2, red[2 B..) = c . x,
// red[3 B..) = b . y (v2rdm_solver.cc:1826-1852), deterministic.
void launch_errors(const DevMap& A, int64_t nx, int64_t nc, int B, const double* aty, const double* x, const double* y,
                   const double* z, const double* c, const double* brow, const int* mask, double* partial, double* red,
                   cudaStream_t s);
// out[e * B + b] = row[e] (or 0 when row is null) for the instances with mask[b] set
void launch_set_rows(int64_t n, int B, const double* row, double* out, const int* mask, cudaStream_t s);

// CG pieces (cg_solver.cc:125-177), per instance with cg_active masks.
struct CgScalars {
    double rr, pap, alpha, beta, rrnew, tol;
    double rrmin;  // smallest r.r of this solve
    int active;    // still iterating
    int iter;      // iter_ of the reference
    int step;      // this iteration takes a step (q.q above rounding noise)
    int maxiter;
    int stalled;   // stopped because r.r grew past kCgGrowth * rrmin
};
// A A^T is singular (the constraint rows are dependent), so a right-hand side
// with a component in the null space of A^T above the CG tolerance (rounding
// in A(c - z) and A x) cannot be met: r stalls at that component and CG then
// diverges, with y growing without bound.  In the converging BPSDP runs
// measured, r.r never rose more than ~30x above its running minimum (|r| 5.3x
// in 4,252 CG solves); a rise past this factor stops the instance's CG with
// the current y instead.
constexpr double kCgGrowth = 1e4;
// The CG of a group as map applications with the vector updates in their
// epilogues (maps.cu, EpiCgQ): r = rhs - A q for q = A^T y and its r.r; then
// per iteration the direction q = A^T r + beta q with alpha from q.q, and the
// step p = r + beta p, y += alpha p, r -= alpha A q with the convergence test
// and beta from r.r, counting the instances still iterating into *n_active.
// Instances with cs[b].active == 0 are left alone.  partial holds
// reduce_partial_size(B) doubles.
void launch_cg_start(const DevMap& A, int B, const double* q, const double* rhs, double* r, CgScalars* cs,
                     double* partial, int* n_active, cudaStream_t s);
void launch_cg_direction(const DevMap& AT, int B, const double* r, double* q, CgScalars* cs, double* partial,
                         int* n_active, cudaStream_t s);
void launch_cg_step(const DevMap& A, int B, const double* q, double* y, double* r, double* p, CgScalars* cs,
                    double* partial, int* n_active, cudaStream_t s);
// Sets the WHILE condition h of a device-side CG loop: ++*count, then
// continue while *n_active > 0 and *count < cap.
void launch_cg_while(cudaGraphConditionalHandle h, const int* n_active, int* count, int cap, cudaStream_t s);

// Persistent CG (maps.cu): a whole CG solve of a small group in one
// cooperative launch.  Groups of at most kLoopMaxB instances and kLoopMaxRows
// constraints (n <= 13 with DQG), where launch latency, not bandwidth, bounds
// an iteration; above, two map launches with their reductions are faster
// (B200, us per iteration, persistent / launches: n = 12 one instance 25.6 /
// 29.7, n = 10 eight instances 41.5 / 46.5, n = 14 one instance 43.2 / 39.6,
// n = 20 one instance 131 / 99).
constexpr int kLoopMaxB = 8;
constexpr int64_t kLoopMaxRows = 300000;
bool cg_loop_fits(const DevMap& A, const DevMap& AT, int B);
// CTAs of the cooperative grid on this device (0: no cooperative launch)
int cg_loop_grid(int device);
size_t cg_loop_slots(int grid, int B);
// The whole solve from y, rhs and cs (tol, active, maxiter set): iterates
// until no instance is active or cap iterations; y, r, p, q and cs as the
// launches above leave them, but p where the resident kernel runs, which keeps it
// in registers; *n_active the instances still active, *iters the
// iterations run, *err = 1 if a wait of the grid's exchanges ran out
// (then the results are invalid; *err must be 0 at the launch).  slots holds
// cg_loop_slots(grid, B) words.
cudaError_t launch_cg_loop(const DevMap& A, const DevMap& AT, int B, const double* rhs, double* y, double* r, double* p,
                           double* q, CgScalars* cs, unsigned long long* slots, int* err, int* n_active,
                           int* iters, int cap, int grid, cudaStream_t s);
// CG start extrapolation over [e * B + b]: where mode[b] == 2,
// y <- y + (y - yprev); where mode[b] >= 1, yprev <- y (its value on entry)
void launch_cg_extrapolate(int64_t n, int B, double* y, double* yprev, const int* mode, cudaStream_t s);
// ---- Anderson acceleration of the outer iteration --------------------------
// The state w = (x, z) of one instance is the 2 * nx rows e < nx of x and
// e >= nx of z, interleaved [e * B + b] like every vector; the history holds
// m difference columns dF_j = f_{k+1} - f_k and dG_j = g_{k+1} - g_k (f = g - w,
// g = the iterate the step produced), each 2 * nx * B doubles, column j at
// j * 2 * nx * B.
constexpr int kAndersonMax = 16;
// f = g - w; mode[b] == 2: dF[slot[b]] = f - fprev, dG[slot[b]] = g - gprev and
// dots[(2 j) * B + b] = dF[slot].dF[j], dots[(2 j + 1) * B + b] = dF[j].f for j < m;
// mode[b] >= 1: dots[(2 m) * B + b] = f.f, fprev = f, gprev = g.  partial holds
// aa_partial_size(nx, B, m) doubles; the sums are deterministic.
void launch_aa_update(int64_t nx, int B, int m, const double* x, const double* z, const double* w, double* fprev,
                      double* gprev, double* dF, double* dG, const int* mode, const int* slot, double* partial,
                      double* dots, cudaStream_t s);
int64_t aa_partial_size(int64_t nx, int B, int m);
// (x, z) <- g - sum_j gamma[b * m + j] dG_j for the instances with mix[b] set
// (columns with gamma 0 are not read)
void launch_aa_mix(int64_t nx, int B, int m, double* x, double* z, const double* dG, const double* gamma,
                   const int* mix, cudaStream_t s);

// ---- projection (Update_xz) ----------------------------------------------

// Description of one PSD block of one instance.
struct BlockTask {
    int64_t xoff;   // offset of the block in the (per-instance) primal vector
    int n;          // block dimension
    int inst;       // instance index within the group (for interleaving)
    int64_t woff;   // offset of the padded workspace matrix (large blocks)
    int np;         // padded dimension (multiple of 64, large blocks)
    int nb;         // number of 32-wide column blocks (np / 32)
    int64_t qoff;   // offset of the pair-rotation buffer (large blocks)
    int64_t doff;   // offset of the np-long weight vector (large blocks)
    int64_t toff;   // offset (32-bit words) of the split TF32 operands (tensor-core blocks)
};

// Blocks with n <= 64 (max_n the largest of them): form U, its matrix sign in
// shared memory, x and z (psd_sign.cu).  hint (optional, one word per task, 0 at
// first) carries the number of lift steps that sufficed to the next call.
// beside: the launch shares the GPU with launch_team_sign.
void launch_small_project(const BlockTask* tasks, int ntasks, int max_n, int B, const double* aty, const double* c,
                          double* x, double* z, const double* mu, const int* mask, cudaStream_t s,
                          int* hint = nullptr, bool beside = false);

// Blocks of any size the same way, a team of CTAs per block in one cooperative
// launch.  Entry w of a CTA: its w-th block, its rank in the block's team and the
// team's size (task -1: none).
struct SignTeam {
    int task, rank, size;
    int64_t base;  // of the team's 2 x size partial sums
};
// CTAs of the cooperative grid on this device (0: no cooperative launch)
int sign_grid(int device);
// Teams of all the blocks on the grid; returns the number of waves (teams: waves
// x grid entries, a CTA's blocks in its order) and of partial sums.
int sign_schedule(const std::vector<BlockTask>& tasks, int grid, std::vector<SignTeam>& teams, int64_t& parts);
// x and z of the blocks of active instances.  atol (per task, optional): accept
// a residual |U (1 - X^2)|_F of that size.  S, X, X2 and A are np x np workspaces
// at task.woff; bar one word per task; hint as above; *err = 1 if a team's wait
// ran out (then the results are invalid).
cudaError_t launch_team_sign(const BlockTask* tasks, int ntasks, const SignTeam* teams, int waves, int grid, int B,
                             const double* aty, const double* c, double* x, double* z, const double* mu,
                             const int* mask, const double* atol, double* S, double* X, double* X2, double* A,
                             double* part, unsigned int* bar, int* hint, int* err, cudaStream_t s);

// Large blocks (n > 64), block Jacobi on a padded np x np workspace.
// U = sym(A^T y - c + mu x), zero padded.
void launch_form_u(const BlockTask* tasks, int ntasks, int max_np, int B, const double* aty, const double* c,
                   const double* x, const double* mu, const int* mask, double* Uw, cudaStream_t s);
// W = U (cold start) and V = I
void launch_cold_start(const BlockTask* tasks, int ntasks, int max_np, const double* Uw, double* Ww, double* Vw,
                       const int* bmask, cudaStream_t s);
// batched 64x64-tiled FP64 GEMM on the padded workspaces:
// C = op(A) diag(d) op(B), with d optional.
struct GemmTile {
    int task;   // block task index
    int ti, tj; // tile coordinates
};
void launch_gemm(const BlockTask* tasks, const GemmTile* tiles, int ntiles, const double* A, bool transA,
                 const double* Bm, bool transB, const double* dvec, double* C, const int* bmask, cudaStream_t s);
// The same product on the tensor cores (tcgen05, 3xTF32 split, FP32
// accumulation: FP32 accuracy) over 128 x 128 tiles of C: tile (ti, tj)
// covers rows 128 ti.. and columns 128 tj..; rows and columns past np are not
// written.  The operands are first split into TF32 pairs in the MMA's shared
// memory layout, one unit (task, 128-row block) per CTA, into the plan's
// workspaces wa and wb (tc_split_words(np) words per task, at task.toff).
struct TcSplit {
    int task, rb;
};
struct TcPlan {
    const BlockTask* tasks = nullptr;
    const GemmTile* tiles_full = nullptr;  // every 128 x 128 tile
    const GemmTile* tiles_sym = nullptr;   // tiles ti <= tj (symmetric products, mirrored afterwards)
    int n_full = 0, n_sym = 0;
    const TcSplit* split = nullptr;
    int nsplit = 0;
    int max_nk = 0;  // largest np / 32 of the tasks: the split runs one CTA per (row block, K chunk)
    uint32_t* wa = nullptr;
    uint32_t* wb = nullptr;
};
int64_t tc_split_words(int np);
void launch_tc_gemm(const TcPlan& plan, bool sym, const double* A, bool transA, const double* Bm, bool transB,
                    const double* dvec, double* C, const int* bmask, cudaStream_t s);
// 0 while every tensor-core GEMM's pipeline waits ended; 1 after one ran out
// (that launch's result is invalid); reset clears the flag.
int tc_gemm_status(bool reset);
// the same flag copied into host (pinned) memory on a stream, without a device-wide sync
void tc_gemm_status_async(int* host, cudaStream_t s);
// One block-Jacobi round: solve each 64x64 pair problem, then rotate W and V.
struct PairTask {
    int task;   // block task
    int k;      // pair index within the round
};
struct WTileTask {
    int task, k1, k2;
};
struct VTileTask {
    int task, chunk, k;
};
// One round of the block Jacobi: each 64x64 pair problem is diagonalised
// into Qbuf unless its off-diagonal norm^2 is at most pthr[task] (then
// qskip marks its rotation as the identity and the update leaves it out).
void launch_bj_solve(const BlockTask* tasks, const PairTask* pt, int npt, int round, double* Ww, double* Qbuf,
                     const int* bmask, const double* pthr, int* qskip, cudaStream_t s);
void launch_bj_update_wv(const BlockTask* tasks, const WTileTask* wt, int nwt, const VTileTask* vt, int nvt, int round,
                         double* Ww, double* Vw, const double* Qbuf, const int* bmask, const int* qskip,
                         cudaStream_t s);
// Per-block off-diagonal and total Frobenius norms of W; sets bmask[t] = 0
// for blocks whose off-diagonal norm is below max(tol[t] * total, abs_tol[t])
// or that have done max_sweeps[t] sweeps, and pthr[t] = that limit squared
// over the pair problems of a sweep.
void launch_bj_check(const BlockTask* tasks, int ntasks, int max_np, const double* Ww, const double* tol,
                     const double* abs_tol, const int* max_sweeps, int sweeps_done, double* rowsum, int* bmask,
                     double* pthr, int* n_open, cudaStream_t s);
// dx = max(lam, 0) / mu and dz = max(-lam, 0) (per block, length np; zero on padding)
void launch_pos_weights(const BlockTask* tasks, int ntasks, const double* lam, const double* mu, const int* bmask,
                        double* dx, double* dz, cudaStream_t s);
// lam = diag(W)
void launch_lam_from_diag(const BlockTask* tasks, int ntasks, const double* Ww, const int* bmask, double* lam,
                          cudaStream_t s);
// Ogita-Aishima step: lam_i = s_ii / g_ii and M = I + E from S = V^T U V and
// G = V^T V; emax[t] gets max |E_ij| (as the bits of a non-negative double)
// and hard[t] is set for blocks needing the Jacobi fallback (an index
// strongly coupled to more than one other; isolated strongly coupled pairs
// are rotated exactly).  partner needs one int per padded row.
// Blocks whose eigenvectors lost orthonormality (|g_ii - 1| > 0.25) or whose
// values broke down get restart[t] = 1; blocks whose first-order step has
// ||E||_F > 0.2 are marked hard.  erow holds one double per padded row.
// gdev[t] (optional) gets max |G_ij - delta_ij| of the block (as the bits of a
// non-negative double): the distance of V from orthonormal.
void launch_oa_analyze(const BlockTask* tasks, int ntasks, int max_np, const double* S, const double* G,
                       const int* bmask, double* lam, double* scale, int* partner, double* M,
                       unsigned long long* emax, int* hard, double* erow, int* restart, unsigned long long* gdev,
                       cudaStream_t s);
void launch_oa_masks(int ntasks, const unsigned long long* emax, const int* hard, const double* tol,
                     const double* abs_tol, const double* scale, int* ref, int* upd, int* jac, int* n_ref,
                     cudaStream_t s);
void launch_copy_blocks(const BlockTask* tasks, int ntasks, int max_np, const double* src, double* dst,
                        const int* bmask, cudaStream_t s);
void launch_count(int n, const int* mask, int* out, cudaStream_t s);
// symmetric GEMM results: copy the upper tiles onto the lower ones
void launch_mirror(const BlockTask* tasks, int ntasks, int max_np, double* C, const int* bmask, cudaStream_t s);
// M = I + (I - G) / 2 (G = V^T V): V M is a Newton-Schulz step that brings V
// back to orthonormal (the distance squares)
void launch_ortho_step(const BlockTask* tasks, int ntasks, int max_np, const double* G, const int* bmask, double* M,
                       cudaStream_t s);
// bmask[t] = mask[tasks[t].inst] != 0
void launch_block_mask(const BlockTask* tasks, int ntasks, const int* mask, int* bmask, cudaStream_t s);
// max_sweeps[i] = unlimited where sel[i]
void launch_uncap(int n, const int* sel, int* max_sweeps, cudaStream_t s);
// dst[i] |= src[i]
void launch_merge_mask(int n, const int* src, int* dst, cudaStream_t s);
// x = X and z = Z (unpadded, interleaved)
void launch_write_xz(const BlockTask* tasks, int ntasks, int max_n, int B, const double* Xw, const double* Zw,
                     const int* mask, double* x, double* z, cudaStream_t s);

}  // namespace v2g
