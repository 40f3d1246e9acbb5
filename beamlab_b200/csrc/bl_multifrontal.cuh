// The multifrontal factorization and solves of the frames' implicit step in two launches (the plan: bl_mf_plan.cuh).
//
// Each front is a lower triangle of 48 x 48 tiles (8 frame nodes a side): its pivots in P tiles, then its rows, the right
// side b one more row after them (so that eliminating the pivots leaves, in b's row, the forward substitution's y on the
// pivots and the update vector of the rows). A tile's 2,304 doubles lie in the order in which the fp64 tensor-core
// instruction (mma.m8n8k4) takes either operand of L L^T: three chunks of 16 columns, each of 8 x 4 blocks whose 32
// entries are a warp's lanes - operand loads from shared memory are conflict-free and a chunk is one contiguous copy.
//
// k_mf_factor and k_mf_back run persistent CTAs over a list of tasks in an order in which every task's inputs come from tasks before
// it: a CTA takes the next task, waits on the flags of what it reads, and sets its own. The earliest unfinished task is
// always held by a running CTA with all its inputs done, so the waits end; each is bounded in time all the same
// (kMfWaitNs, then DEVERR_TIMEOUT, every component marked failed, the CTAs leave).
//   tile (f, i, j)   the tile's assembled blocks, its children's Schur complements in the children's order (extend-add),
//                    less sum_k L_ik L_jk^T over the pivot panels k before j (left-looking: the sum stays in the tensor
//                    cores' accumulators, L tiles stream through a ring of asynchronous copies as they become ready);
//                    then for a pivot column j: the diagonal tile is factored and its inverse kept, a tile below it is
//                    multiplied by that inverse; a tile past the pivots is the Schur complement its parent takes.
//   front (f)        a front of one pivot tile and up to three row tiles, b's among them, in a wide level (most leaves of large
//                    bodies): all its tiles by one CTA, no flags
//   backward (f, s)  from the root down: x_s = L_ss^-T (y_s - sum_(i > s) L_is^T x_i), the rows' x from the ancestors
// No atomics on values and every sum in a fixed order: the same bits every run. rhs gets the solution in column order.
// A pivot that is not positive marks the front's component failed (the reference's chol6 failing, frame_fem.cpp:
// 2900-2909: that component's step falls back to its explicit forces) and goes on as 1.
//
// What bounds it: small frames by the chain of dependent panels (a panel ~12 us: the diagonal tile's inverse factor 4.0, a
// product with it 2.5, the update of the next diagonal tile 2.5, the rest flags and loads through L2; 3.9 on the way back), large
// ones by the tiles' operands from L2 and a barrier a chunk, at 0.27 of the fp64 rate. 48: a multiple of a node's 6 degrees of freedom and of the instruction's 8, three CTAs an SM with both
// operands' ring. Measured on B200 (factorization and solves alone; before: minimum-degree fronts, a launch a panel and
// a launch an update, 32 x 32 tiles on the plain fp64 units): the 21 x 21 plate 0.21 ms, the 64 x 64 plate 0.56 (3.9),
// the 10k-node shell body 1.43 (7.8), the 50k-node one 6.3 (38.0): 63.3 GFLOP at 10.1 TFLOP/s of the 35.5 a cuBLAS
// DGEMM reaches, 24 to 28 in the large fronts.
#pragma once

#include "bl_fem_kernels.cuh"
#include "bl_mf_plan.cuh"

namespace blg {

constexpr int kMfChunk = kMfT * 16;    // doubles a chunk (16 columns)
constexpr int kMfThreads = 128;
constexpr int kMfStages = 4;           // the ring: chunks of both operands in flight
#ifndef BL_MF_WAIT_NS // (a test builds the library with 0: every wait that is not over at once runs out)
#define BL_MF_WAIT_NS 4000000000ull
#endif
constexpr unsigned long long kMfWaitNs = BL_MF_WAIT_NS;
constexpr size_t kMfSmem = sizeof(double) * (2 * kMfStages * kMfChunk + kMfTile);

struct MfDev {
    const MfFrontDev* fr;
    const int* idx;
    const int* cpos;
    const int* cptr;
    const int* child;
    const int* pan;      // per global column: its panel
    const int* eptr;     // per tile + 1: its assembled blocks in ent
    const int2* ent;     // (off-diagonal block, or -(column + 1) for a diagonal one; 8 row slot + column slot)
    double* pool;        // kMfTile a tile
    const int4* task;    // (front, i, j, kind)
    int nfactor, ntask, ncomp; // the factorization's tasks, then the backward solves'
    int* ctr;            // zeroed before each step: [0] the next task, [1] abort, [2] the next backward one, then
    int* fdone;          // per front
    int* tflag;          // per tile
    int* xflag;          // per panel: the backward solve's warps that are done (4)
};
// entry (r, c) of a tile
__host__ __device__ __forceinline__ int mf_at(int r, int c) {
    return (c >> 4) * kMfChunk + (r >> 3) * 128 + ((c >> 2) & 3) * 32 + (r & 7) * 4 + (c & 3);
}
__device__ __forceinline__ int mf_ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mf_st_release(int* p, int v) { asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void mf_add_release(int* p, int v) { asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }

// waits until *p >= target; false when the launch is aborted or the wait runs out (it then aborts the launch)
__device__ __forceinline__ bool mf_wait(const int* p, int target, int* abort_flag) {
    unsigned long long t0 = 0;
    for (int it = 0;; it++) {
        if (mf_ld_acquire(p) >= target) return true;
        if ((it & 63) == 63) {
            if (*(volatile int*)abort_flag) return false;
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t0 == 0) t0 = t;
            if (t - t0 >= kMfWaitNs) {
                atomicExch(abort_flag, 1);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void mf_cp16(double* dst, const double* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void mf_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void mf_cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void mf_copy_chunk(double* dst, const double* src) {
    for (int e = threadIdx.x; e < kMfChunk / 2; e += kMfThreads) mf_cp16(dst + 2 * e, src + 2 * e);
}
__device__ __forceinline__ void mf_mma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// A warp's 3 x 3 blocks of 8 x 8 of a tile: block rows 0, 3, 4 (wr = 0) or 1, 2, 5, block columns likewise by wc - so that the
// four warps share the lower triangle of a diagonal tile (6, 4, 5, 6 blocks) and the columns of a triangular factor
// evenly (a contiguous quarter each: 9 and 3 blocks, 36 and 6 of a column's 8-wide terms).
__device__ __forceinline__ int mf_own(int w, int x) { return w == 0 ? (x == 0 ? 0 : x + 2) : (x == 2 ? 5 : x + 1); }
// acc += A B^T over one chunk (16 of the summed columns). lower: only blocks on and below the diagonal.
template <bool kLower>
__device__ __forceinline__ void mf_mma_chunk(double (&acc)[3][3][2], const double* A, const double* B, int wr, int wc, int lane) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        double a[3], b[3];
#pragma unroll
        for (int x = 0; x < 3; x++) a[x] = A[mf_own(wr, x) * 128 + k * 32 + lane], b[x] = B[mf_own(wc, x) * 128 + k * 32 + lane];
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++)
                if (!kLower || mf_own(wr, x) >= mf_own(wc, y)) mf_mma(acc[x][y], a[x], b[y]);
    }
}
// acc = A B^T of two tiles, B lower triangular
__device__ __forceinline__ void mf_mma_lower(double (&acc)[3][3][2], const double* A, const double* B, int wr, int wc, int lane) {
#pragma unroll 2
    for (int k = 0; k < 12; k++) {
        const int at = (k >> 2) * kMfChunk + (k & 3) * 32 + lane;
        double a[3];
#pragma unroll
        for (int x = 0; x < 3; x++) a[x] = A[at + mf_own(wr, x) * 128];
#pragma unroll
        for (int y = 0; y < 3; y++) {
            if (mf_own(wc, y) < k >> 1) continue;
            const double b = B[at + mf_own(wc, y) * 128];
#pragma unroll
            for (int x = 0; x < 3; x++) mf_mma(acc[x][y], a[x], b);
        }
    }
}
// where this lane's pair of accumulator (x, y) lies in a tile
__device__ __forceinline__ int mf_acc_at(int x, int y, int wr, int wc, int lane) {
    const int c = 8 * mf_own(wc, y) + 2 * (lane & 3);
    return (c >> 4) * kMfChunk + mf_own(wr, x) * 128 + ((c >> 2) & 3) * 32 + (lane >> 2) * 4 + (c & 3);
}

// ---- the diagonal tile's factor and its inverse, in 8 x 8 blocks (64 contiguous doubles of a tile)
__device__ __forceinline__ int mf_blk(int rb, int cb) { return (cb >> 1) * kMfChunk + rb * 128 + (cb & 1) * 64; }
// acc += A B^T and acc += A B of two blocks, by a warp
__device__ __forceinline__ void mf_abt8(double (&acc)[2], const double* A, const double* B, int lane) {
    mf_mma(acc, A[lane], B[lane]);
    mf_mma(acc, A[32 + lane], B[32 + lane]);
}
__device__ __forceinline__ void mf_ab8(double (&acc)[2], const double* A, const double* B, int lane) {
    const int t = (lane >> 4) * 32 + (lane & 3) * 4 + ((lane >> 2) & 3); // (B's entry (lane & 3, lane >> 2))
    mf_mma(acc, A[lane], B[t]);
    mf_mma(acc, A[32 + lane], B[t + 16]);
}
// where this lane's pair of an 8 x 8 accumulator lies in a block
__device__ __forceinline__ int mf_pair8(int lane) { return ((lane & 3) >> 1) * 32 + (lane >> 2) * 4 + 2 * (lane & 1); }

// The inverse of an 8 x 8 block's Cholesky factor, by one warp: every lane factors the block in its own registers, so
// that a column's chain is the inverse square root, a multiply and a multiply-add with no exchange of lanes; lane i < 8
// carries row i of an identity along, which comes out as column i of the inverse. (Lanes a row each and the columns
// broadcast by shuffles: 190 cycles a column against 85.) False at a pivot that is not positive or not finite.
__device__ __forceinline__ bool mf_inv8(const double* B, double* inv, int lane) {
    double d[8][8], a[8];
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
        for (int c = 0; c <= r; c += 2) {
            const double2 u = *reinterpret_cast<const double2*>(B + (c >> 2) * 32 + r * 4 + (c & 3));
            d[r][c] = u.x, d[r][c + 1] = u.y;
        }
#pragma unroll
    for (int c = 0; c < 8; c++) a[c] = c == lane ? 1.0 : 0.0;
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const double id = bl_pivot_rsqrt(d[j][j], ok);
        if (j == 7) ok = ok && id == id; // (an infinite pivot: no number from it on, so the next pivot says so, or this)
#pragma unroll
        for (int l = j + 1; l < 8; l++) d[l][j] *= id;
        a[j] *= id;
#pragma unroll
        for (int l = j + 1; l < 8; l++) {
#pragma unroll
            for (int m = j + 1; m <= l; m++) d[l][m] = fma(-d[l][j], d[m][j], d[l][m]);
            a[l] = fma(-a[j], d[l][j], a[l]);
        }
    }
    if (lane < 8)
#pragma unroll
        for (int r = 0; r < 8; r++) inv[(lane >> 2) * 32 + r * 4 + (lane & 3)] = r >= lane ? a[r] : 0.0;
    return ok;
}

// The transposed inverse X of the diagonal tile's Cholesky factor (upper; zero before); D (lower) is overwritten by the
// factor's blocks below the diagonal. The identity is carried as six more block rows below the tile: eliminating the
// tile's columns turns it into the transposed inverse. By columns of 8: the first warp makes the chain -
// L_(k+1)k = D_(k+1)k inv_k^T, the next diagonal block less L L^T, its factor's inverse inv_(k+1) - while the other
// three make the rest of the block column (always six blocks) and its updates of the later blocks, evenly. One
// barrier a column of blocks. The chain bounds it: 48 columns of an inverse square root, a multiply and a
// multiply-add. scr: 2 blocks of inverses in turn, the chain's L. False at a pivot that is not positive.
// (9.6 us with panels of 16 columns, plain multiply-adds for the updates and the inverse after them; 5.3 with the
// inverse's rows made one after the other.)
constexpr int kMfScr = 3 * 64;
__device__ __forceinline__ bool mf_factor_tile(double* D, double* X, double* scr, int* bad) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = warp - 1, pr = mf_pair8(lane);
    double *inv = scr, *Lc = scr + 2 * 64;
    auto at2 = [&](double* p) -> double2& { return *reinterpret_cast<double2*>(p + pr); };
    if (warp == 0 && !mf_inv8(D, inv, lane) && lane == 0) *bad = 1;
    __syncthreads();
    for (int kb = 0; kb < 6; kb++) {
        const double* ik = inv + 64 * (kb & 1);
        if (warp == 0) {
            if (kb < 5) {
                double* N = D + mf_blk(kb + 1, kb + 1);
                double t[2] = {0.0, 0.0}, u[2] = {0.0, 0.0};
                mf_abt8(t, D + mf_blk(kb + 1, kb), ik, lane);
                at2(Lc) = make_double2(t[0], t[1]); // (the chain's own copy: another warp stores L for the rest)
                asm volatile("bar.arrive 2, 128;" ::: "memory");
                __syncwarp();
                mf_abt8(u, Lc, Lc, lane);
                at2(N) = make_double2(at2(N).x - u[0], at2(N).y - u[1]);
                __syncwarp();
                if (!mf_inv8(N, inv + 64 * ((kb + 1) & 1), lane) && lane == 0) *bad = 1;
            }
        } else {
            // the block column: the tile's rows kb + 1 .. 5, then the identity's 0 .. kb; two blocks a warp
            double t[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
            double* row[2]; // (the block row's first block; its others lie mf_blk(0, c) from it)
            int last[2];    // its last block column to update
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const int q = w + 3 * x, i = q - (5 - kb);
                row[x] = (i < 0 ? D : X) + mf_blk(i < 0 ? kb + 1 + q : i, 0);
                last[x] = i >= 0 ? 5 : q == 0 ? kb : kb + 1 + q; // (row kb + 1's one block is the chain's)
                double a0 = (lane >> 2) == (lane & 3) ? 1.0 : 0.0, a1 = (lane >> 2) == (lane & 3) + 4 ? 1.0 : 0.0; // (the identity's own block)
                if (i != kb) a0 = row[x][mf_blk(0, kb) + lane], a1 = row[x][mf_blk(0, kb) + 32 + lane];
                mf_mma(t[x], a0, ik[lane]), mf_mma(t[x], a1, ik[32 + lane]);
            }
            // (the chain reads D_(k+1)k too, at the start of this step: its copy is made before this one is stored)
            if (kb < 5) asm volatile("bar.sync 2, 128;" ::: "memory");
            else __syncwarp();
#pragma unroll
            for (int x = 0; x < 2; x++) at2(row[x] + mf_blk(0, kb)) = make_double2(t[x][0], t[x][1]);
            asm volatile("bar.sync 1, 96;" ::: "memory"); // (the three warps: the block column is there)
            // the later blocks of these two rows less their product with the block column (a loop of few instructions:
            // unrolled over its blocks it waited for its code)
            double a[2][2];
#pragma unroll
            for (int x = 0; x < 2; x++) a[x][0] = -row[x][mf_blk(0, kb) + lane], a[x][1] = -row[x][mf_blk(0, kb) + 32 + lane];
#pragma unroll 1
            for (int cb = kb + 1; cb < 6; cb++) {
                const double* L = D + mf_blk(cb, kb);
                const double b0 = L[lane], b1 = L[32 + lane];
#pragma unroll
                for (int x = 0; x < 2; x++) {
                    if (cb > last[x]) continue;
                    double2 d = at2(row[x] + mf_blk(0, cb));
                    double v[2] = {d.x, d.y};
                    mf_mma(v, a[x][0], b0), mf_mma(v, a[x][1], b1);
                    at2(row[x] + mf_blk(0, cb)) = make_double2(v[0], v[1]);
                }
            }
        }
        __syncthreads();
    }
    return *bad == 0;
}

// The tile's assembled blocks and its children's Schur complements into C (shared). The children's maps - which of a
// child's row nodes falls on each of the tile's 8 row and 8 column slots - are made before they are waited for; then a
// thread gathers three rows of six entries each, over the children in their order. False when the launch aborts.
constexpr int kMfKids = 16; // children at a time (8 threads each)
struct MfKids {
    int base[kMfKids], nt[kMfKids], P[kMfKids], bt[kMfKids], br[kMfKids]; // first tile, tiles a side, pivot tiles, b's tile and row
    int row[kMfKids][8], col[kMfKids][8];                                 // its row node on each slot, -1: none
};
__device__ __forceinline__ bool mf_assemble(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int i, int j, double* C, MfKids& K) {
    const int tid = threadIdx.x;
    for (int e = tid; e < kMfTile / 2; e += kMfThreads) reinterpret_cast<double2*>(C)[e] = make_double2(0.0, 0.0);
    __syncthreads();
    if (j < fr.P) {
        const int t = fr.tile0 + mf_tix(fr.nt, i, j), e0 = M.eptr[t], e1 = M.eptr[t + 1];
        for (int e = tid; e < 18 * (e1 - e0); e += kMfThreads) { // (a thread a pair of a block's entries)
            const int2 s = M.ent[e0 + e / 18];
            const int x = 2 * (e % 18), a = x / 6, b = x % 6;
            const double* B = s.x >= 0 ? F.off + 36 * (size_t)s.x : F.diag + 36 * (size_t)(-s.x - 1);
            *reinterpret_cast<double2*>(C + mf_at(6 * (s.y >> 3) + a, 6 * (s.y & 7) + b)) = *reinterpret_cast<const double2*>(B + x);
        }
        if (i == fr.bt && tid < kMfT && 8 * j + tid / 6 < fr.npiv) C[mf_at(fr.br, tid)] = F.rhs[6 * (size_t)M.idx[fr.idx0 + 8 * j + tid / 6] + tid % 6];
        if (i == j && tid < kMfT && kMfT * j + tid >= fr.p) C[mf_at(tid, tid)] = 1.0; // (past the last pivot: an identity)
    }
    for (int q0 = fr.child0; q0 < fr.child1; q0 += kMfKids) {
        const int nq = min(kMfKids, fr.child1 - q0), q = tid >> 3, k = tid & 7;
        if (q0 > fr.child0) __syncthreads(); // (the maps' readers are done)
        bool ok = true;
        if (q < nq) {
            const int c = M.child[q0 + q];
            const MfFrontDev& cf = M.fr[c];
            const int* cp = M.cptr + cf.cptr0;
            const int* pos = M.cpos + cf.cpos0;
            const int rx = cp[i] + k, re = cp[i + 1], cx = cp[j] + k, ce = cp[j + 1];
            const int rp = rx < re ? pos[rx] : -1, cq = cx < ce ? pos[cx] : -1;
            if (k == 0) K.base[q] = cf.tile0, K.nt[q] = cf.nt, K.P[q] = cf.P, K.bt[q] = cf.bt, K.br[q] = cf.br;
            K.row[q][k] = -1, K.col[q][k] = -1;
            __syncwarp(0xffu << (tid & 24)); // (the child's eight threads: q < nq holds for all of them or none)
            if (rp >= 0) K.row[q][rp & 7] = rx;
            if (cq >= 0) K.col[q][cq & 7] = cx;
            if (k == 0) ok = mf_wait(M.fdone + c, cf.need, M.ctr + 1);
        }
        if (__syncthreads_or(!ok)) return false;
        double2 v[3][3];
        bool any[3] = {false, false, false};
#pragma unroll
        for (int m = 0; m < 3; m++)
#pragma unroll
            for (int b = 0; b < 3; b++) v[m][b] = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int c = 0; c < nq; c++) {
            const double* S = M.pool + (size_t)K.base[c] * kMfTile;
            const int nt = K.nt[c], P = K.P[c];
            double2 u[3][3];
            bool on[3];
#pragma unroll
            for (int m = 0; m < 3; m++) { // (row a of the node pair (dr, dc))
                const int g = tid + kMfThreads * m, pair = g / 6, a = g - 6 * pair, qr = K.row[c][pair >> 3], qc = K.col[c][pair & 7];
                on[m] = qr >= qc && qc >= 0;
                if (!on[m]) continue;
                any[m] = true;
                const double* T = S + (size_t)mf_tix(nt, P + (qr >> 3), P + (qc >> 3)) * kMfTile;
#pragma unroll
                for (int b = 0; b < 3; b++) u[m][b] = __ldcg(reinterpret_cast<const double2*>(T + mf_at(6 * (qr & 7) + a, 6 * (qc & 7) + 2 * b)));
            }
#pragma unroll
            for (int m = 0; m < 3; m++)
                if (on[m])
#pragma unroll
                    for (int b = 0; b < 3; b++) v[m][b].x += u[m][b].x, v[m][b].y += u[m][b].y;
        }
#pragma unroll
        for (int m = 0; m < 3; m++) {
            if (!any[m]) continue;
            const int g = tid + kMfThreads * m, pair = g / 6, a = g - 6 * pair;
#pragma unroll
            for (int b = 0; b < 3; b++) {
                double2* d = reinterpret_cast<double2*>(C + mf_at(6 * (pair >> 3) + a, 6 * (pair & 7) + 2 * b));
                const double2 o = *d;
                *d = make_double2(o.x + v[m][b].x, o.y + v[m][b].y);
            }
        }
        if (i == fr.bt && tid < kMfT) { // (b's row)
            double t = 0;
            for (int c = 0; c < nq; c++) {
                const int qc = K.col[c][tid / 6];
                if (qc >= 0)
                    t += __ldcg(M.pool + (size_t)(K.base[c] + mf_tix(K.nt[c], K.bt[c], K.P[c] + (qc >> 3))) * kMfTile + mf_at(K.br[c], 6 * (qc & 7) + tid % 6));
            }
            C[mf_at(fr.br, tid)] += t;
        }
    }
    __syncthreads();
    return true;
}

// One tile of a front (alone: by this CTA alone, its inputs of the same front written by this CTA before)
__device__ __forceinline__ bool mf_tile(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int f, int i, int j, bool alone, double* ring, double* C) {
    __shared__ int s_ready, s_bad;
    __shared__ MfKids s_kids;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 1, wc = warp >> 1;
    if (!mf_assemble(F, M, fr, i, j, C, s_kids)) return false;
    const double* base = M.pool + (size_t)fr.tile0 * kMfTile;
    double acc[3][3][2];
#pragma unroll
    for (int x = 0; x < 3; x++)
#pragma unroll
        for (int y = 0; y < 3; y++) acc[x][y][0] = acc[x][y][1] = 0.0;
    const int nk = min(j, fr.P);
    const bool same = i == j;
    for (int k0 = 0; k0 < nk;) {
        int k1 = nk;
        if (!alone) {
            // the panels ready from k0 on (at least one: waited for), by the first warp's lanes
            if (warp == 0) {
                bool ok = mf_wait(M.tflag + fr.tile0 + mf_tix(fr.nt, i, k0), 1, M.ctr + 1) &&
                          (same || mf_wait(M.tflag + fr.tile0 + mf_tix(fr.nt, j, k0), 1, M.ctr + 1));
                const int k = k0 + lane;
                const bool r = ok && k < nk && mf_ld_acquire(M.tflag + fr.tile0 + mf_tix(fr.nt, i, k)) &&
                               (same || mf_ld_acquire(M.tflag + fr.tile0 + mf_tix(fr.nt, j, k)));
                const unsigned m = __ballot_sync(0xffffffffu, r);
                if (lane == 0) s_ready = k0 + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
            }
            __syncthreads();
            k1 = s_ready;
            if (k1 <= k0) return false;
        }
        const int nch = 3 * (k1 - k0);
        auto issue = [&](int c) {
            if (c < nch) {
                const int k = k0 + c / 3, kc = c % 3, st = c % kMfStages;
                mf_copy_chunk(ring + 2 * st * kMfChunk, base + (size_t)mf_tix(fr.nt, i, k) * kMfTile + kc * kMfChunk);
                if (!same) mf_copy_chunk(ring + (2 * st + 1) * kMfChunk, base + (size_t)mf_tix(fr.nt, j, k) * kMfTile + kc * kMfChunk);
            }
            mf_cp_commit();
        };
#pragma unroll
        for (int c = 0; c < kMfStages - 1; c++) issue(c);
        for (int c = 0; c < nch; c++) {
            mf_cp_wait<kMfStages - 2>();
            __syncthreads();
            issue(c + kMfStages - 1);
            const double* A = ring + 2 * (c % kMfStages) * kMfChunk;
            if (same) mf_mma_chunk<true>(acc, A, A, wr, wc, lane);
            else mf_mma_chunk<false>(acc, A, A + kMfChunk, wr, wc, lane);
        }
        mf_cp_wait<0>();
        __syncthreads();
        k0 = k1;
    }
    double* out = M.pool + (size_t)(fr.tile0 + mf_tix(fr.nt, i, j)) * kMfTile;
    if (j >= fr.P) { // the Schur complement
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++) {
                const int at = mf_acc_at(x, y, wr, wc, lane);
                const double2 c = *reinterpret_cast<const double2*>(C + at);
                *reinterpret_cast<double2*>(out + at) = make_double2(c.x - acc[x][y][0], c.y - acc[x][y][1]);
            }
        __syncthreads();
        if (!alone && tid == 0) mf_add_release(M.fdone + f, 1);
        return true;
    }
    if (same) {
        double* X = ring;
        if (tid == 0) s_bad = 0;
        for (int e = tid; e < kMfTile / 2; e += kMfThreads) reinterpret_cast<double2*>(X)[e] = make_double2(0.0, 0.0);
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++) {
                double2* c = reinterpret_cast<double2*>(C + mf_acc_at(x, y, wr, wc, lane));
                *c = make_double2(c->x - acc[x][y][0], c->y - acc[x][y][1]);
            }
        __syncthreads();
        const bool ok = mf_factor_tile(C, X, ring + kMfTile, &s_bad);
        for (int e = tid; e < kMfTile / 2; e += kMfThreads) { // (the inverse: X transposed; the pair e of the tile's order)
            const int kc = e / (kMfChunk / 2), q = e % (kMfChunk / 2), rb = q / 64, cb = (q / 16) & 3, l = 2 * (q & 15);
            const int r = 8 * rb + l / 4, c = 16 * kc + 4 * cb + l % 4;
            reinterpret_cast<double2*>(out)[e] = make_double2(X[mf_at(c, r)], X[mf_at(c + 1, r)]);
        }
        if (!ok && tid == 0) atomicExch(&F.comp_fail[fr.comp], 1);
    } else {
        // X = A L_jj^-T
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++) {
                const int at = mf_acc_at(x, y, wr, wc, lane);
                const double2 c = *reinterpret_cast<const double2*>(C + at);
                *reinterpret_cast<double2*>(C + at) = make_double2(c.x - acc[x][y][0], c.y - acc[x][y][1]);
                acc[x][y][0] = acc[x][y][1] = 0.0;
            }
        const int dt = mf_tix(fr.nt, j, j);
        bool ok = true;
        if (!alone && tid == 0) ok = mf_wait(M.tflag + fr.tile0 + dt, 1, M.ctr + 1);
        if (__syncthreads_or(!ok)) return false;
        for (int kc = 0; kc < 3; kc++) mf_copy_chunk(ring + kc * kMfChunk, base + (size_t)dt * kMfTile + kc * kMfChunk);
        mf_cp_commit();
        mf_cp_wait<0>();
        __syncthreads();
        mf_mma_lower(acc, C, ring, wr, wc, lane);
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++)
                *reinterpret_cast<double2*>(out + mf_acc_at(x, y, wr, wc, lane)) = make_double2(acc[x][y][0], acc[x][y][1]);
    }
    __syncthreads();
    if (!alone && tid == 0) mf_st_release(M.tflag + fr.tile0 + mf_tix(fr.nt, i, j), 1);
    return true;
}

// a tile's 18 entries of this lane for the products with its transpose: columns 4 cb + (lane & 3), cb = warp + 4 m, rows
// 8 rb + lane / 4
__device__ __forceinline__ void mf_load_cols(double (&v)[3][6], const double* T, int warp, int lane) {
#pragma unroll
    for (int m = 0; m < 3; m++)
#pragma unroll
        for (int rb = 0; rb < 6; rb++) v[m][rb] = __ldcg(T + m * kMfChunk + rb * 128 + warp * 32 + lane);
}
__device__ __forceinline__ void mf_dot_cols(double (&acc)[3], const double (&v)[3][6], const double* x, int lane) {
#pragma unroll
    for (int rb = 0; rb < 6; rb++) {
        const double xr = x[8 * rb + (lane >> 2)];
#pragma unroll
        for (int m = 0; m < 3; m++) acc[m] = fma(v[m][rb], xr, acc[m]);
    }
}
__device__ __forceinline__ double mf_sum_rows(double t) {
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    return t + __shfl_xor_sync(0xffffffffu, t, 16);
}

// x of a front's panel s: its rows' x (its ancestors') as they become known - the highest first, up to kMfXTiles tiles at a
// time, each group when the panel of its lowest node is solved (then all above it are) - then its own later panels', then
// x_s = L_ss^-T z. A warp that has stored its part of x_s adds one to the panel's flag.
constexpr int kMfXTiles = 8;
__device__ __forceinline__ bool mf_backward(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int s, double* xs, double* z) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* base = M.pool + (size_t)fr.tile0 * kMfTile;
    const int* idx = M.idx + fr.idx0;
    double acc[3] = {0, 0, 0}, v[3][6];
    double y[3]; // (this lane's of the panel's y)
#pragma unroll
    for (int m = 0; m < 3; m++) y[m] = __ldcg(base + (size_t)mf_tix(fr.nt, fr.bt, s) * kMfTile + mf_at(fr.br, 4 * (warp + 4 * m) + (lane & 3)));
    bool ok = true;
    for (int t1 = (fr.nrow + 7) / 8; t1 > 0; t1 -= kMfXTiles) {
        const int t0 = max(0, t1 - kMfXTiles), nt = t1 - t0;
        const double* L = base + (size_t)mf_tix(fr.nt, fr.P + t0, s) * kMfTile; // (a column's tiles lie one after the other)
        mf_load_cols(v, L, warp, lane);                                      // (before the wait)
        int at[kMfXTiles * kMfT / kMfThreads];
#pragma unroll
        for (int x = 0; x < kMfXTiles * kMfT / kMfThreads; x++) {
            const int e = tid + kMfThreads * x, q = 8 * t0 + e / 6;
            at[x] = e < nt * kMfT && q < fr.nrow ? 6 * idx[fr.npiv + q] + e % 6 : -1;
        }
        if (ok) ok = mf_wait(M.xflag + M.pan[idx[fr.npiv + 8 * t0]], 4, M.ctr + 1);
#pragma unroll
        for (int x = 0; x < kMfXTiles * kMfT / kMfThreads; x++) xs[tid + kMfThreads * x] = at[x] >= 0 ? __ldcg(F.rhs + at[x]) : 0.0;
        if (__syncthreads_or(!ok)) return false;
        for (int t = 0; t < nt; t++) {
            double w[3][6];
            if (t + 1 < nt) mf_load_cols(w, L + (size_t)(t + 1) * kMfTile, warp, lane);
            mf_dot_cols(acc, v, xs + t * kMfT, lane);
#pragma unroll
            for (int m = 0; m < 3; m++)
#pragma unroll
                for (int rb = 0; rb < 6; rb++) v[m][rb] = w[m][rb];
        }
        __syncthreads();
    }
    for (int i = fr.P - 1; i > s; i--) {
        mf_load_cols(v, base + (size_t)mf_tix(fr.nt, i, s) * kMfTile, warp, lane); // (before the wait)
        if (tid < kMfT) {
            const int at = kMfT * i + tid < fr.p ? 6 * idx[8 * i + tid / 6] + tid % 6 : -1;
            ok = mf_wait(M.xflag + fr.pan0 + i, 4, M.ctr + 1);
            xs[(i & 1) * kMfT + tid] = at >= 0 ? __ldcg(F.rhs + at) : 0.0;
        }
        if (__syncthreads_or(!ok)) return false;
        mf_dot_cols(acc, v, xs + (i & 1) * kMfT, lane);
    }
    mf_load_cols(v, base + (size_t)mf_tix(fr.nt, s, s) * kMfTile, warp, lane); // (L_ss^-1)
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const double t = mf_sum_rows(acc[m]);
        const int c = 4 * (warp + 4 * m) + lane;
        if (lane < 4) z[c] = y[m] - t;
        acc[m] = 0.0;
    }
    __syncthreads();
    mf_dot_cols(acc, v, z, lane);
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const double t = mf_sum_rows(acc[m]);
        const int c = kMfT * s + 4 * (warp + 4 * m) + lane;
        if (lane < 4 && c < fr.p) F.rhs[6 * (size_t)idx[c / 6] + c % 6] = t;
    }
    __syncwarp();
    if (lane == 0) mf_add_release(M.xflag + fr.pan0 + s, 1);
    __syncthreads(); // (xs, z: the next task's)
    return true;
}

// the launch was aborted: flagged, every component failed
__device__ __forceinline__ void mf_leave(const FemDev& F, const MfDev& M, uint32_t* deverr) {
    if (!*(volatile int*)(M.ctr + 1)) return;
    if (threadIdx.x == 0) atomicOr(deverr, DEVERR_TIMEOUT);
    for (int c = threadIdx.x; c < M.ncomp; c += kMfThreads) F.comp_fail[c] = 1;
}

// The factorization: 128 threads, 66 KB of shared memory, three CTAs an SM
__global__ void __launch_bounds__(kMfThreads, 3) k_mf_factor(FemDev F, MfDev M, uint32_t* deverr) {
    extern __shared__ __align__(16) double mf_smem[];
    __shared__ int s_task;
    double* ring = mf_smem;
    double* C = mf_smem + 2 * kMfStages * kMfChunk;
    for (;;) {
        if (threadIdx.x == 0) s_task = *(volatile int*)(M.ctr + 1) ? -1 : atomicAdd(M.ctr, 1);
        __syncthreads();
        const int t = s_task;
        __syncthreads();
        if (t < 0 || t >= M.nfactor) break;
        const int4 task = M.task[t];
        const MfFrontDev fr = M.fr[task.x];
        // one tile, or all of a front's (a root's Schur complement is nobody's)
        const bool alone = task.w == MF_FRONT;
        const int j1 = !alone ? task.z + 1 : fr.parent >= 0 ? fr.nt : fr.P;
        bool ok = true;
#pragma unroll 1
        for (int j = task.z; ok && j < j1; j++) {
            const int i1 = alone ? fr.nt : task.y + 1;
#pragma unroll 1
            for (int i = alone ? j : task.y; ok && i < i1; i++) {
                ok = mf_tile(F, M, fr, task.x, i, j, alone, ring, C);
                if (alone) __syncthreads();
            }
        }
        if (alone && ok && threadIdx.x == 0) mf_add_release(M.fdone + task.x, 1);
        if (!ok) break;
    }
    mf_leave(F, M, deverr);
}

// The backward solves, after it
__global__ void __launch_bounds__(kMfThreads, 3) k_mf_back(FemDev F, MfDev M, uint32_t* deverr) {
    __shared__ double xs[kMfXTiles * kMfT], z[kMfT];
    __shared__ int s_task;
    for (;;) {
        if (threadIdx.x == 0) s_task = *(volatile int*)(M.ctr + 1) ? -1 : M.nfactor + atomicAdd(M.ctr + 2, 1);
        __syncthreads();
        const int t = s_task;
        __syncthreads();
        if (t < 0 || t >= M.ntask) break;
        const int4 task = M.task[t];
        if (!mf_backward(F, M, M.fr[task.x], task.z, xs, z)) break;
    }
    mf_leave(F, M, deverr);
}

} // namespace blg
