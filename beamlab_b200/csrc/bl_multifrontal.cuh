// The multifrontal factorization and solves of the frames' implicit step in one launch (the plan: bl_mf_plan.cuh).
//
// Each front is a lower triangle of 48 x 48 tiles (8 frame nodes a side): its pivots in P tiles, then its rows, the right
// side b one more row after them (so that eliminating the pivots leaves, in b's row, the forward substitution's y on the
// pivots and the update vector of the rows). A tile's 2,304 doubles lie in the order in which the fp64 tensor-core
// instruction (mma.m8n8k4) takes either operand of L L^T: three chunks of 16 columns, each of 8 x 4 blocks whose 32
// entries are a warp's lanes - operand loads from shared memory are conflict-free and a chunk is one contiguous copy.
//
// k_mf_solve runs persistent CTAs over one list of tasks in an order in which every task's inputs come from tasks before
// it: a CTA takes the next task, waits on the flags of what it reads, and sets its own. The earliest unfinished task is
// always held by a running CTA with all its inputs done, so the waits end; each is bounded in time all the same
// (kMfWaitNs, then DEVERR_TIMEOUT, every component marked failed, the CTAs leave).
//   tile (f, i, j)   the tile's assembled blocks, its children's Schur complements in the children's order (extend-add),
//                    less sum_k L_ik L_jk^T over the pivot panels k before j (left-looking: the sum stays in the tensor
//                    cores' accumulators, L tiles stream through a ring of asynchronous copies as they become ready);
//                    then for a pivot column j: the diagonal tile is factored and its inverse kept, a tile below it is
//                    multiplied by that inverse; a tile past the pivots is the Schur complement its parent takes.
//   front (f)        a front of one pivot tile and at most two row tiles (most leaves): all its tiles by one CTA, no flags
//   backward (f, s)  from the root down: x_s = L_ss^-T (y_s - sum_(i > s) L_is^T x_i), the rows' x from the ancestors
// No atomics on values and every sum in a fixed order: the same bits every run. rhs gets the solution in column order.
// A pivot that is not positive marks the front's component failed (the reference's chol6 failing, frame_fem.cpp:
// 2900-2909: that component's step falls back to its explicit forces) and goes on as 1.
//
// What bounds it: small frames by the chain of dependent panels (a panel ~16 us: the diagonal tile's 48 dependent columns
// and inverse 10, a product with its inverse 2.5, the update of the next diagonal tile 2.5, their flags 1 each), large
// ones by the fp64 rate. 48: a multiple of a node's 6 degrees of freedom and of the instruction's 8, three CTAs an SM
// with both operands' ring. Measured on B200 (factorization and solves alone; before: the same fronts with a launch a
// panel and a launch an update, 32 x 32 tiles on the plain fp64 units): the 64 x 64 plate 1.07 ms (3.9), the 10k-node
// shell body 2.0 (7.8), the 50k-node one 8.8 (38.0: 82.9 GFLOP at 9.4 TFLOP/s of the 35.5 a cuBLAS DGEMM reaches).
#pragma once

#include "bl_fem_kernels.cuh"
#include "bl_mf_plan.cuh"

namespace blg {

constexpr int kMfChunk = kMfT * 16;    // doubles a chunk (16 columns)
constexpr int kMfThreads = 128;
constexpr int kMfStages = 4;           // the ring: chunks of both operands in flight
constexpr unsigned long long kMfWaitNs = 4000000000ull;
constexpr size_t kMfSmem = sizeof(double) * (2 * kMfStages * kMfChunk + kMfTile);

struct MfDev {
    const MfFrontDev* fr;
    const int* idx;
    const int* cpos;
    const int* cptr;
    const int* child;
    const int* eptr;     // per tile + 1: its assembled blocks in ent
    const int2* ent;     // (off-diagonal block, or -(column + 1) for a diagonal one; 8 row slot + column slot)
    double* pool;        // kMfTile a tile
    const int4* task;    // (front, i, j, kind)
    int ntask, ncomp;
    int* ctr;            // zeroed before each launch: [0] the next task, [1] abort, then
    int* fdone;          // per front
    int* xdone;          // per front: panels solved backward
    int* tflag;          // per tile
    int* xflag;          // per panel
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
            else if (t - t0 > kMfWaitNs) {
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

// acc += A B^T over one chunk (16 of the summed columns): a warp's 24 x 24 quarter of the tile, 3 x 3 blocks of 8 x 8
__device__ __forceinline__ void mf_mma_chunk(double (&acc)[3][3][2], const double* A, const double* B, int wr, int wc, int lane) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        double a[3], b[3];
#pragma unroll
        for (int x = 0; x < 3; x++) a[x] = A[(3 * wr + x) * 128 + k * 32 + lane], b[x] = B[(3 * wc + x) * 128 + k * 32 + lane];
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++) mf_mma(acc[x][y], a[x], b[y]);
    }
}
// where this lane's pair of accumulator (x, y) lies in a tile
__device__ __forceinline__ int mf_acc_at(int x, int y, int wr, int wc, int lane) {
    const int c = 8 * (3 * wc + y) + 2 * (lane & 3);
    return (c >> 4) * kMfChunk + (3 * wr + x) * 128 + ((c >> 2) & 3) * 32 + (lane >> 2) * 4 + (c & 3);
}

constexpr int kMfLd = kMfT + 1; // the plain layout of the diagonal tile's factorization

// A panel of 16 columns (c0 ..) of the diagonal tile, rows c0 .. 47, by one warp: lane l holds row c0 + l and, where there
// is one, row c0 + l + 32. A column's chain is its pivot's broadcast, the inverse square root, a multiply and the next
// pivot's update, which its own lane makes from its own entry; the other columns' updates read the finished column
// from shared memory meanwhile.
__device__ __forceinline__ bool mf_panel16(double (*D)[kMfLd], int c0, int lane) {
    double a0[16], a1[16];
    const int r0 = c0 + lane, r1 = c0 + lane + 32;
    const bool h0 = r0 < kMfT, h1 = r1 < kMfT;
#pragma unroll
    for (int j = 0; j < 16; j++) a0[j] = h0 ? D[r0][c0 + j] : 0.0, a1[j] = h1 ? D[r1][c0 + j] : 0.0;
    bool ok = true;
    double piv = a0[0];
#pragma unroll
    for (int j = 0; j < 16; j++) {
        double s = __shfl_sync(0xffffffffu, piv, j);
        if (!(s > 0)) ok = false, s = 1.0;
        const double id = rsqrt(s);
        a0[j] = lane == j ? s * id : a0[j] * id;
        a1[j] *= id;
        if (j < 15) piv = fma(-a0[j], a0[j], a0[j + 1]); // (lane j + 1's next pivot)
        if (h0) D[r0][c0 + j] = lane >= j ? a0[j] : 0.0;
        if (h1) D[r1][c0 + j] = a1[j];
        if (lane == j) D[r0][kMfT] = id; // (the pad column: the pivots' inverses)
        __syncwarp();
#pragma unroll
        for (int l = j + 1; l < 16; l++) {
            const double t = D[c0 + l][c0 + j];
            a0[l] = fma(-a0[j], t, a0[l]), a1[l] = fma(-a1[j], t, a1[l]);
        }
    }
    return ok;
}

// The inverse of the 16 x 16 lower triangle at c0, by one warp (lane c < 16: column c), into Y
__device__ __forceinline__ void mf_inv16(double (*D)[kMfLd], double (*Y)[kMfLd], int c0, int lane) {
    if (lane >= 16) return;
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; r++) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
    for (int r = 0; r < 16; r++) {
        x[r] *= D[c0 + r][kMfT];
#pragma unroll
        for (int q = r + 1; q < 16; q++) x[q] = fma(-D[c0 + q][c0 + r], x[r], x[q]);
    }
#pragma unroll
    for (int r = 0; r < 16; r++) Y[c0 + r][c0 + lane] = x[r];
}

// Z (16 x 16 at zr, zc) = s A (ar, ac) B (br, bc), by the whole block, two entries a thread
__device__ __forceinline__ void mf_mul16(double (*Z)[kMfLd], int zr, int zc, double (*A)[kMfLd], int ar, int ac, double (*B)[kMfLd], int br, int bc,
                                         double s, bool add) {
    const int r = threadIdx.x >> 3, c = threadIdx.x & 7;
    double t0 = 0, t1 = 0;
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const double a = A[ar + r][ac + m];
        t0 = fma(a, B[br + m][bc + c], t0), t1 = fma(a, B[br + m][bc + c + 8], t1);
    }
    if (add) t0 = fma(s, t0, Z[zr + r][zc + c]), t1 = fma(s, t1, Z[zr + r][zc + c + 8]);
    else t0 *= s, t1 *= s;
    Z[zr + r][zc + c] = t0, Z[zr + r][zc + c + 8] = t1;
}

// The diagonal tile's Cholesky factor and the factor's inverse: D (plain, lower) in, Y out. Three panels of 16 columns by
// the first warp, each followed by the block's update of the columns after it while the second warp inverts the
// panel's triangle; then the inverse's blocks below the diagonal. False at a pivot that is not positive.
__device__ __forceinline__ bool mf_factor_tile(double (*D)[kMfLd], double (*Y)[kMfLd], int* bad) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int kb = 0; kb < 3; kb++) {
        const int c0 = 16 * kb;
        if (warp == 0) {
            if (!mf_panel16(D, c0, lane) && lane == 0) *bad = 1;
        } else if (kb > 0 && warp == 1) {
            mf_inv16(D, Y, c0 - 16, lane);
        }
        __syncthreads();
        // the columns after the panel, lower triangle: D_rc -= sum_m L_rm L_cm, 8 (2) entries a thread
        if (kb == 0) {
            const int r = 16 + (tid >> 2), q = tid & 3; // (row r; columns 16 + q + 4 x)
            double t[8];
#pragma unroll
            for (int x = 0; x < 8; x++) t[x] = 0;
#pragma unroll
            for (int m = 0; m < 16; m++) {
                const double l = D[r][m];
#pragma unroll
                for (int x = 0; x < 8; x++) t[x] = fma(l, D[16 + q + 4 * x][m], t[x]);
            }
#pragma unroll
            for (int x = 0; x < 8; x++)
                if (16 + q + 4 * x <= r) D[r][16 + q + 4 * x] -= t[x];
        } else if (kb == 1) {
            const int r = 32 + (tid >> 3), q = tid & 7;
            double t0 = 0, t1 = 0;
#pragma unroll
            for (int m = 16; m < 32; m++) t0 = fma(D[r][m], D[32 + q][m], t0), t1 = fma(D[r][m], D[40 + q][m], t1);
            if (32 + q <= r) D[r][32 + q] -= t0;
            if (40 + q <= r) D[r][40 + q] -= t1;
        }
        if (kb < 2) __syncthreads();
    }
    // the inverse: Y00, Y11 there, Y22 now; T = L10 Y00, Y10 = -Y11 T; U = L20 Y00 + L21 Y10, W = L21 Y11;
    // Y20 = -Y22 U, Y21 = -Y22 W (T, U, W in D's upper blocks (0, 1), (0, 2), (1, 2))
    if (warp == 3) mf_inv16(D, Y, 32, lane);
    mf_mul16(D, 0, 16, D, 16, 0, Y, 0, 0, 1.0, false);
    mf_mul16(D, 0, 32, D, 32, 0, Y, 0, 0, 1.0, false);
    mf_mul16(D, 16, 32, D, 32, 16, Y, 16, 16, 1.0, false);
    __syncthreads();
    mf_mul16(Y, 16, 0, Y, 16, 16, D, 0, 16, -1.0, false);
    mf_mul16(Y, 32, 16, Y, 32, 32, D, 16, 32, -1.0, false);
    __syncthreads();
    mf_mul16(D, 0, 32, D, 32, 16, Y, 16, 0, 1.0, true);
    __syncthreads();
    mf_mul16(Y, 32, 0, Y, 32, 32, D, 0, 32, -1.0, false);
    __syncthreads();
    return *bad == 0;
}

// The tile's assembled blocks and its children's contributions into C (shared, zeroed). False when the launch aborts.
__device__ __forceinline__ bool mf_assemble(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int i, int j, double* C) {
    const int tid = threadIdx.x;
    for (int e = tid; e < kMfTile / 2; e += kMfThreads) reinterpret_cast<double2*>(C)[e] = make_double2(0.0, 0.0);
    bool ok = true;
    for (int q = fr.child0 + tid; q < fr.child1; q += kMfThreads) {
        const int c = M.child[q];
        ok = ok && mf_wait(M.fdone + c, M.fr[c].need, M.ctr + 1);
    }
    if (__syncthreads_or(!ok)) return false;
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
    for (int q = fr.child0; q < fr.child1; q++) {
        const MfFrontDev cf = M.fr[M.child[q]];
        const int* cp = M.cptr + cf.cptr0;
        const int* pos = M.cpos + cf.cpos0;
        const int ra = cp[i], rb = cp[i + 1], ca = cp[j], nc = cp[j + 1] - ca;
        if (nc == 0 || (ra == rb && i != fr.bt)) continue;
        __syncthreads();
        const double* S = M.pool + (size_t)cf.tile0 * kMfTile;
        for (int e = tid; e < 6 * (rb - ra) * nc; e += kMfThreads) {
            const int qc = ca + e % nc, t = e / nc, a = t % 6, qr = ra + t / 6;
            if (qr < qc) continue;
            const double* T = S + (size_t)mf_tix(cf.nt, cf.P + (qr >> 3), cf.P + (qc >> 3)) * kMfTile;
            const int sr = 6 * (qr & 7) + a, sc = 6 * (qc & 7), dr = 6 * (pos[qr] & 7) + a, dc = 6 * (pos[qc] & 7);
            double2 v[3];
#pragma unroll
            for (int b = 0; b < 3; b++) v[b] = __ldcg(reinterpret_cast<const double2*>(T + mf_at(sr, sc + 2 * b)));
#pragma unroll
            for (int b = 0; b < 3; b++) {
                double2* d = reinterpret_cast<double2*>(C + mf_at(dr, dc + 2 * b));
                const double2 o = *d;
                *d = make_double2(o.x + v[b].x, o.y + v[b].y);
            }
        }
        if (i == fr.bt)
            for (int e = tid; e < 6 * nc; e += kMfThreads) {
                const int qc = ca + e / 6;
                const double* T = S + (size_t)mf_tix(cf.nt, cf.bt, cf.P + (qc >> 3)) * kMfTile;
                C[mf_at(fr.br, 6 * (pos[qc] & 7) + e % 6)] += __ldcg(T + mf_at(cf.br, 6 * (qc & 7) + e % 6));
            }
    }
    __syncthreads();
    return true;
}

// One tile of a front (alone: by this CTA alone, its inputs of the same front written by this CTA before)
__device__ bool mf_tile(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int f, int i, int j, bool alone, double* ring, double* C) {
    __shared__ int s_ready, s_bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 1, wc = warp >> 1;
    if (!mf_assemble(F, M, fr, i, j, C)) return false;
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
            mf_mma_chunk(acc, A, same ? A : A + kMfChunk, wr, wc, lane);
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
        double(*D)[kMfLd] = reinterpret_cast<double(*)[kMfLd]>(ring);
        double(*Y)[kMfLd] = D + kMfT;
        if (tid == 0) s_bad = 0;
#pragma unroll
        for (int x = 0; x < 3; x++)
#pragma unroll
            for (int y = 0; y < 3; y++) {
                const double2 c = *reinterpret_cast<const double2*>(C + mf_acc_at(x, y, wr, wc, lane));
                const int r = 8 * (3 * wr + x) + (lane >> 2), cc = 8 * (3 * wc + y) + 2 * (lane & 3);
                D[r][cc] = c.x - acc[x][y][0], D[r][cc + 1] = c.y - acc[x][y][1];
            }
        for (int e = tid; e < kMfT * kMfLd; e += kMfThreads) (&Y[0][0])[e] = 0.0;
        __syncthreads();
        const bool ok = mf_factor_tile(D, Y, &s_bad);
        for (int e = tid; e < kMfTile / 2; e += kMfThreads) { // (the pair e of the tile's order)
            const int kc = e / (kMfChunk / 2), q = e % (kMfChunk / 2), rb = q / 64, cb = (q / 16) & 3, l = 2 * (q & 15);
            const int r = 8 * rb + l / 4, c = 16 * kc + 4 * cb + l % 4;
            reinterpret_cast<double2*>(out)[e] = make_double2(Y[r][c], Y[r][c + 1]);
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
        for (int kc = 0; kc < 3; kc++) mf_mma_chunk(acc, C + kc * kMfChunk, ring + kc * kMfChunk, wr, wc, lane);
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

// x of a front's panel s, from its rows' x (its ancestors') and its later panels'
constexpr int kMfXTiles = 96; // row tiles' x held at a time
__device__ bool mf_backward(const FemDev& F, const MfDev& M, const MfFrontDev& fr, int f, int s, double* ring) {
    double* xs = ring;                       // kMfXTiles x 48
    double* z = ring + kMfXTiles * kMfT;     // 48
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* base = M.pool + (size_t)fr.tile0 * kMfTile;
    const int* idx = M.idx + fr.idx0;
    double acc[3] = {0, 0, 0}, li[3][6], v[3][6];
    // its tiles: a root's by their flags; below, the parent's solution comes after the whole factorization of both
    bool ok = true;
    if (fr.parent < 0) {
        for (int i = s + tid; i < fr.nt; i += kMfThreads) ok = ok && mf_wait(M.tflag + fr.tile0 + mf_tix(fr.nt, i, s), 1, M.ctr + 1);
    } else if (tid == 0) {
        ok = mf_wait(M.xdone + fr.parent, M.fr[fr.parent].P, M.ctr + 1);
    }
    if (__syncthreads_or(!ok)) return false;
    mf_load_cols(li, base + (size_t)mf_tix(fr.nt, s, s) * kMfTile, warp, lane);
    const double y = tid < kMfT ? __ldcg(base + (size_t)mf_tix(fr.nt, fr.bt, s) * kMfTile + mf_at(fr.br, tid)) : 0.0;
    if (fr.nrow > 0) {
        const int nrt = (fr.nrow + 7) / 8;
        for (int t0 = 0; t0 < nrt; t0 += kMfXTiles) {
            const int nt = min(kMfXTiles, nrt - t0);
            if (t0 > 0) __syncthreads();
            for (int e = tid; e < nt * kMfT; e += kMfThreads) {
                const int q = 8 * t0 + e / 6;
                xs[e] = q < fr.nrow ? __ldcg(F.rhs + 6 * (size_t)idx[fr.npiv + q] + e % 6) : 0.0;
            }
            __syncthreads();
            for (int t = 0; t < nt; t++) {
                mf_load_cols(v, base + (size_t)mf_tix(fr.nt, fr.P + t0 + t, s) * kMfTile, warp, lane);
                mf_dot_cols(acc, v, xs + t * kMfT, lane);
            }
        }
    }
    for (int i = fr.P - 1; i > s; i--) {
        mf_load_cols(v, base + (size_t)mf_tix(fr.nt, i, s) * kMfTile, warp, lane); // (before the wait)
        if (tid == 0) ok = mf_wait(M.xflag + fr.pan0 + i, 1, M.ctr + 1);
        if (__syncthreads_or(!ok)) return false;
        if (tid < kMfT) xs[tid] = kMfT * i + tid < fr.p ? __ldcg(F.rhs + 6 * (size_t)idx[8 * i + tid / 6] + tid % 6) : 0.0;
        __syncthreads();
        mf_dot_cols(acc, v, xs, lane);
    }
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const double t = mf_sum_rows(acc[m]);
        if (lane < 4) z[4 * (warp + 4 * m) + lane] = t;
        acc[m] = 0.0;
    }
    __syncthreads();
    if (tid < kMfT) z[tid] = y - z[tid];
    __syncthreads();
    mf_dot_cols(acc, li, z, lane);
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const double t = mf_sum_rows(acc[m]);
        const int c = kMfT * s + 4 * (warp + 4 * m) + lane;
        if (lane < 4 && c < fr.p) F.rhs[6 * (size_t)idx[c / 6] + c % 6] = t;
    }
    __syncthreads();
    if (tid == 0) mf_st_release(M.xflag + fr.pan0 + s, 1), mf_add_release(M.xdone + f, 1);
    return true;
}

// 128 threads, 66 KB of shared memory: three CTAs an SM
__global__ void __launch_bounds__(kMfThreads, 3) k_mf_solve(FemDev F, MfDev M, uint32_t* deverr) {
    extern __shared__ __align__(16) double mf_smem[];
    __shared__ int s_task;
    double* ring = mf_smem;
    double* C = mf_smem + 2 * kMfStages * kMfChunk;
    for (;;) {
        if (threadIdx.x == 0) s_task = *(volatile int*)(M.ctr + 1) ? -1 : atomicAdd(M.ctr, 1);
        __syncthreads();
        const int t = s_task;
        __syncthreads();
        if (t < 0 || t >= M.ntask) break;
        const int4 task = M.task[t];
        const MfFrontDev fr = M.fr[task.x];
        bool ok = true;
        if (task.w == MF_TILE) {
            ok = mf_tile(F, M, fr, task.x, task.y, task.z, false, ring, C);
        } else if (task.w == MF_BACK) {
            ok = mf_backward(F, M, fr, task.x, task.z, ring);
        } else {
            const int last = fr.parent >= 0 ? fr.nt : fr.P; // (a root's Schur complement is nobody's)
            for (int j = 0; ok && j < last; j++)
                for (int i = j; ok && i < fr.nt; i++) {
                    ok = mf_tile(F, M, fr, task.x, i, j, true, ring, C);
                    __syncthreads();
                }
            if (ok && threadIdx.x == 0) {
                for (int k = 0; k < fr.nt; k++) mf_st_release(M.tflag + fr.tile0 + k, 1); // (its one pivot column's)
                mf_add_release(M.fdone + task.x, 1);
            }
        }
        if (!ok) break;
    }
    if (*(volatile int*)(M.ctr + 1)) {
        if (threadIdx.x == 0) atomicOr(deverr, DEVERR_TIMEOUT);
        for (int c = threadIdx.x; c < M.ncomp; c += kMfThreads) F.comp_fail[c] = 1;
    }
}

} // namespace blg
