// Host side of the multifrontal factorization of a frame's implicit step (the kernels: bl_multifrontal.cuh).
//
// The reference factors the step's block system column by column, right-looking, with the exact minimum-degree order
// of its symbolic phase (frame_fem.cpp:2887-2920). Here the columns come in a nested-dissection order (FemDissection,
// bl_fem_host.cuh) and are grouped into fronts: dense blocks factored with dense kernels, which is where a GPU is fast.
//  * Elimination tree: column k's parent is its first off-diagonal row.
//  * Fundamental supernodes: a column joins its parent's group when it is that parent's only child and its rows are the
//    parent and the parent's rows (the columns then share one dense structure).
//  * Relaxed amalgamation: a group merges into its parent group while the merged group stays small or adds few
//    explicit zeros (the thresholds below, in frame nodes: 6 degrees of freedom each).
//  * Each front holds its pivots (its columns) and its rows (the structure above them), both in elimination order, as
//    a lower triangle of 48 x 48 tiles, the pivots in tiles of their own. Its factorization eliminates the pivots and
//    leaves the Schur complement of its rows in place, which its parent adds into its own front (extend-add).
//  * The tiles are tasks in one list - fronts by level of the front tree, leaves first, a level's tiles column by column -
//    in which every task's inputs come before it (mf_layout).
// The solution equals the column-by-column one up to the order of the floating-point sums.
#pragma once

#include <vector_functions.h>
#include <vector_types.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define MF_HD __host__ __device__ __forceinline__
#else
#define MF_HD inline
#endif

namespace blg {

struct MfPlan {
    // per front, in execution order (by level, leaves first)
    std::vector<int> npiv, nrow;    // frame nodes
    std::vector<int> parent;        // front, -1 at a root
    std::vector<int> idx_ptr, idx;  // the front's nodes (global columns: pivots then rows), ascending
    std::vector<int> cmap;          // per front, at idx_ptr + npiv: its rows' places in its parent's node list
    std::vector<int> child_ptr, child;
    std::vector<int> level_ptr;     // fronts of level L: [level_ptr[L], level_ptr[L + 1])
    std::vector<int> comp;          // the component each front belongs to (global)
    double flops = 0;               // per factorization (multiply and add counted apart)
    int chain = 0;                  // the most pivot tiles of 8 nodes (panels) from a leaf to its root
    double entries = 0;             // dense lower-triangle entries over all fronts (DOF^2 / 2)
};

struct MfParams { // relaxed amalgamation, in frame nodes (CHOLMOD's rule of thumb, scaled to 6 x 6 blocks)
    int small = 2;        // merged groups up to this many columns merge whatever their zeros
    int mid = 8;          // ... up to this many, while zeros stay under mid_frac of the entries
    double mid_frac = 0.5;
    int large = 24;
    double large_frac = 0.1;
    double huge_frac = 0.05;
};

// the columns [0, n) of the pattern col_ptr / row (rows ascending; comp_of_col: each column's component): the fronts'
// columns, their top columns and components appended to fr_cols / fr_top / fr_comp
static void mf_plan_columns(int n, const std::vector<int>& col_ptr, const std::vector<int>& row, const std::vector<int>& comp_of_col,
                            std::vector<std::vector<int>>& fr_cols, std::vector<int>& fr_top, std::vector<int>& fr_comp,
                            const MfParams& prm = MfParams{}) {
    std::vector<int> parent(n, -1), nchild(n, 0), only_child(n, -1);
    for (int k = 0; k < n; k++)
        if (col_ptr[k + 1] > col_ptr[k]) {
            parent[k] = row[col_ptr[k]];
            nchild[parent[k]]++, only_child[parent[k]] = k;
        }
    // fundamental supernodes: groups of columns, each in ascending order
    std::vector<int> group(n, -1);
    std::vector<std::vector<int>> cols;
    std::vector<int> top; // the group's last column (its structure is the group's rows)
    for (int k = 0; k < n; k++) {
        const int c = only_child[k];
        const bool chain = nchild[k] == 1 && (col_ptr[c + 1] - col_ptr[c]) == (col_ptr[k + 1] - col_ptr[k]) + 1;
        if (chain) {
            group[k] = group[c];
            cols[group[k]].push_back(k);
            top[group[k]] = k;
        } else {
            group[k] = (int)cols.size();
            cols.push_back({k});
            top.push_back(k);
        }
    }
    const int G = (int)cols.size();
    // the group tree; groups in order of their top column come children before parents
    std::vector<int> gpar(G, -1);
    for (int g = 0; g < G; g++)
        if (parent[top[g]] >= 0) gpar[g] = group[parent[top[g]]];
    std::vector<int> gorder(G);
    for (int g = 0; g < G; g++) gorder[g] = g;
    std::sort(gorder.begin(), gorder.end(), [&](int a, int b) { return top[a] < top[b]; });
    // relaxed amalgamation: zeros[g] / entries[g] over the group's columns in the front it would form
    std::vector<double> zeros(G, 0.0), entries(G, 0.0);
    std::vector<int> alive(G, 1), merged_into(G, -1);
    auto nrows = [&](int g) { return col_ptr[top[g] + 1] - col_ptr[top[g]]; };
    for (int g = 0; g < G; g++) {
        const double m = (double)cols[g].size(), r = nrows(g);
        entries[g] = m * (m + 1) / 2 + m * r;
    }
    auto root_of = [&](int g) {
        while (merged_into[g] >= 0) g = merged_into[g];
        return g;
    };
    for (int gi = 0; gi < G; gi++) {
        const int s = gorder[gi];
        if (gpar[s] < 0) continue;
        const int p = root_of(gpar[s]);
        const double ms = (double)cols[s].size(), mp = (double)cols[p].size(), rp = nrows(p), rs = nrows(s);
        // S's columns in the merged front reach P's columns and rows instead of their own rows
        const double added = ms * (mp + rp - rs);
        const double z = zeros[s] + zeros[p] + added, e = entries[s] + entries[p] + added;
        const double mm = ms + mp, frac = z / e;
        const bool take = mm <= prm.small || (mm <= prm.mid && frac < prm.mid_frac) || (mm <= prm.large && frac < prm.large_frac) || frac < prm.huge_frac;
        if (!take) continue;
        for (int k : cols[s]) cols[p].push_back(k);
        std::vector<int>().swap(cols[s]);
        zeros[p] = z, entries[p] = e;
        alive[s] = 0, merged_into[s] = p;
    }
    for (int g = 0; g < G; g++) {
        if (!alive[g]) continue;
        std::sort(cols[g].begin(), cols[g].end());
        fr_cols.push_back(cols[g]);
        fr_top.push_back(top[g]);
        fr_comp.push_back(comp_of_col[cols[g][0]]);
    }
}

// the fronts (their columns) into the plan: rows, tree, levels, maps
static MfPlan mf_finish(int NF, const std::vector<int>& col_ptr, const std::vector<int>& row, const std::vector<std::vector<int>>& fr_cols,
                        const std::vector<int>& fr_top, const std::vector<int>& fr_comp) {
    MfPlan P;
    const int nfr = (int)fr_cols.size();
    std::vector<int> front_of(NF, -1);
    for (int f = 0; f < nfr; f++)
        for (int k : fr_cols[f]) front_of[k] = f;
    std::vector<int> fpar(nfr, -1), lvl(nfr, 0);
    for (int f = 0; f < nfr; f++) {
        const int t = fr_top[f];
        if (col_ptr[t + 1] > col_ptr[t]) fpar[f] = front_of[row[col_ptr[t]]];
    }
    // levels: a front one above its highest child (children have lower top columns: one pass in top order)
    std::vector<int> order(nfr);
    for (int f = 0; f < nfr; f++) order[f] = f;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return fr_top[a] < fr_top[b]; });
    for (int f : order)
        if (fpar[f] >= 0) lvl[fpar[f]] = std::max(lvl[fpar[f]], lvl[f] + 1);
    int nlev = 0;
    for (int f = 0; f < nfr; f++) nlev = std::max(nlev, lvl[f] + 1);
    // execution order: by level, then by size (largest first, so the long blocks start early), then by top column
    std::vector<int> ex(nfr);
    for (int f = 0; f < nfr; f++) ex[f] = f;
    auto rows_of = [&](int f) { return col_ptr[fr_top[f] + 1] - col_ptr[fr_top[f]]; };
    std::sort(ex.begin(), ex.end(), [&](int a, int b) {
        if (lvl[a] != lvl[b]) return lvl[a] < lvl[b];
        const int sa = (int)fr_cols[a].size() + rows_of(a), sb = (int)fr_cols[b].size() + rows_of(b);
        if (sa != sb) return sa > sb;
        return fr_top[a] < fr_top[b];
    });
    std::vector<int> pos(nfr);
    for (int i = 0; i < nfr; i++) pos[ex[i]] = i;
    P.level_ptr.assign(nlev + 1, 0);
    for (int f = 0; f < nfr; f++) P.level_ptr[lvl[f] + 1]++;
    for (int L = 0; L < nlev; L++) P.level_ptr[L + 1] += P.level_ptr[L];
    P.idx_ptr.assign(1, 0);
    for (int i = 0; i < nfr; i++) {
        const int f = ex[i];
        const int t = fr_top[f];
        P.npiv.push_back((int)fr_cols[f].size());
        P.nrow.push_back(col_ptr[t + 1] - col_ptr[t]);
        P.parent.push_back(fpar[f] >= 0 ? pos[fpar[f]] : -1);
        P.comp.push_back(fr_comp[f]);
        P.idx.insert(P.idx.end(), fr_cols[f].begin(), fr_cols[f].end());
        P.idx.insert(P.idx.end(), row.begin() + col_ptr[t], row.begin() + col_ptr[t + 1]);
        P.idx_ptr.push_back((int)P.idx.size());
        const double p = 6.0 * P.npiv.back(), r = 6.0 * P.nrow.back();
        P.flops += p * p * p / 3 + p * p * r + p * r * r;
        P.entries += (p + r) * (p + r + 1) / 2;
    }
    std::vector<int> chain(nfr, 0);
    for (int f = 0; f < nfr; f++) { // (children first)
        P.chain = std::max(P.chain, chain[f] += (P.npiv[f] + 7) / 8);
        if (P.parent[f] >= 0) chain[P.parent[f]] = std::max(chain[P.parent[f]], chain[f]);
    }
    // each front's rows in its parent's node list (both ascending: one merge walk)
    P.cmap.assign(P.idx.size(), -1);
    for (int f = 0; f < nfr; f++) {
        const int q = P.parent[f];
        if (q < 0) continue;
        int a = P.idx_ptr[q];
        for (int x = P.idx_ptr[f] + P.npiv[f]; x < P.idx_ptr[f + 1]; x++) {
            while (a < P.idx_ptr[q + 1] && P.idx[a] < P.idx[x]) a++;
            P.cmap[x] = a - P.idx_ptr[q]; // (always found: a front's rows are in its parent's list)
        }
    }
    // children in execution order
    std::vector<std::vector<int>> ch(nfr);
    for (int f = 0; f < nfr; f++)
        if (P.parent[f] >= 0) ch[P.parent[f]].push_back(f);
    P.child_ptr.assign(1, 0);
    for (int f = 0; f < nfr; f++) {
        P.child.insert(P.child.end(), ch[f].begin(), ch[f].end());
        P.child_ptr.push_back((int)P.child.size());
    }
    return P;
}

// ------------------------------------------------------------------------------------------ the device's tiles and tasks
constexpr int kMfT = 48;               // tile side (8 frame nodes)
constexpr int kMfTile = kMfT * kMfT;   // doubles a tile
// In a level of many tasks (over kMfWide: several rounds of all resident CTAs) a front of one pivot tile and up to
// kMfFuseRows row tiles is one task: no flags, its tiles still in the cache. In a narrower level its tiles are tasks of
// their own, side by side. (B200, ms a substep with the line at 0, 1,000, 3,000, 10,000 and no whole fronts: the 41 x 41 plate
// 0.51, 0.41 and so on; 64 x 64 0.69, 0.65, 0.62, 0.62, 0.62; 91 x 91 1.03, 1.03, 1.05, 1.05, 1.05; shell bodies of 5,000 nodes
// 1.02, 1.02, 0.97, 0.97, 0.97; 10,000 1.53, 1.52, 1.55, 1.58, 1.58; 20,000 2.64, 2.64, 2.64, 2.78, 2.79; 50,000 6.66, 6.65,
// 6.65, 6.65, 7.03.)
constexpr int kMfFuseRows = 3, kMfWide = 3000;

struct MfFrontDev {
    int p, npiv, nrow;   // pivot degrees of freedom, pivot and row nodes
    int P, nt;           // pivot tiles, tiles a side
    int bt, br;          // b's row tile, its row in it
    int tile0;           // its first tile (column by column of the lower triangle)
    int idx0;            // its nodes (global columns: pivots, then rows) in idx
    int cpos0, cptr0;    // its row nodes' places in its parent (8 tile + slot) in cpos; per parent tile its first row node
    int child0, child1;
    int parent, comp;
    int need;            // what fdone reaches when its Schur complement is complete
    int pan0;            // its panels' flags in xflag
};

enum : int { MF_TILE = 0, MF_FRONT = 1, MF_BACK = 2 };

// tile (i, j), i >= j, of a front of nt tiles a side
MF_HD int mf_tix(int nt, int i, int j) { return j * nt - j * (j - 1) / 2 + (i - j); }

struct MfLayout {
    std::vector<MfFrontDev> fr;
    std::vector<int> cpos, cptr, eptr, pan; // (MfDev's arrays)
    std::vector<int2> ent;
    std::vector<int4> task;
    int64_t tiles = -1;                 // over all fronts (-1: more than fit their indexes)
    int pans = 0;                       // pivot tiles on the diagonals
    int nfactor = 0;                    // the factorization's tasks; the backward solves' come after
    int widest = 1, widest_back = 1;    // the most of either in one level
};

// The plan's tiles, maps and task list for k_mf_factor and k_mf_back; goff_ptr: the off-diagonal blocks' assembly entries (a block
// without any is fill, zero before the factorization)
static MfLayout mf_layout(const MfPlan& P, const std::vector<int>& col_ptr, const std::vector<int>& row, const std::vector<int>& goff_ptr) {
    MfLayout Y;
    const int nfr = (int)P.npiv.size(), nlev = (int)P.level_ptr.size() - 1;
    std::vector<MfFrontDev>& fr = Y.fr;
    fr.resize(nfr);
    int64_t tiles = 0;
    int pans = 0;
    std::vector<int> level(nfr), tasks(nlev, 0);
    auto alone = [&](int f) { return tasks[level[f]] > kMfWide && fr[f].P == 1 && fr[f].nt - fr[f].P <= kMfFuseRows; };
    for (int L = 0; L < nlev; L++)
        for (int f = P.level_ptr[L]; f < P.level_ptr[L + 1]; f++) {
            const int nt = (P.npiv[f] + 7) / 8 + P.nrow[f] / 8 + 1;
            level[f] = L, tasks[L] += nt * (nt + 1) / 2;
        }
    for (int f = 0; f < nfr; f++) {
        MfFrontDev& d = fr[f];
        d.npiv = P.npiv[f], d.nrow = P.nrow[f], d.p = 6 * d.npiv;
        d.P = (d.npiv + 7) / 8;
        d.nt = d.P + d.nrow / 8 + 1; // (the rows and b's row after them)
        d.bt = d.P + d.nrow / 8, d.br = 6 * (d.nrow % 8);
        d.idx0 = P.idx_ptr[f], d.child0 = P.child_ptr[f], d.child1 = P.child_ptr[f + 1], d.parent = P.parent[f], d.comp = P.comp[f];
        d.tile0 = (int)tiles, d.pan0 = pans;
        tiles += (int64_t)d.nt * (d.nt + 1) / 2, pans += d.P;
        const int R = d.nt - d.P;
        d.need = alone(f) ? 1 : d.parent >= 0 ? R * (R + 1) / 2 : 1;
    }
    if (tiles > (int64_t)1 << 30) return Y; // (its tiles' indexes; such a pool is far past the GPU's memory)
    Y.tiles = tiles, Y.pans = pans;
    Y.pan.assign(col_ptr.size() - 1, 0);
    for (int f = 0; f < nfr; f++)
        for (int l = 0; l < fr[f].npiv; l++) Y.pan[P.idx[fr[f].idx0 + l]] = fr[f].pan0 + l / 8;
    // each row node's place in its parent's tiles, and per parent tile a front's first row node
    std::vector<int>&cpos = Y.cpos, &cptr = Y.cptr;
    for (int f = 0; f < nfr; f++) {
        MfFrontDev& d = fr[f];
        d.cpos0 = (int)cpos.size(), d.cptr0 = (int)cptr.size();
        if (d.parent < 0) continue;
        const MfFrontDev& q = fr[d.parent];
        const int* place = P.cmap.data() + d.idx0 + d.npiv;
        int t = 0;
        for (int x = 0; x < d.nrow; x++) {
            const int l = place[x], pos = l < q.npiv ? l : 8 * q.P + (l - q.npiv);
            for (; t <= pos / 8; t++) cptr.push_back(x);
            cpos.push_back(pos);
        }
        for (; t <= q.nt; t++) cptr.push_back(d.nrow);
    }
    // each pivot tile's assembled blocks (those with entries: the fill's are zero)
    std::vector<int>& eptr = Y.eptr;
    std::vector<int2>& ent = Y.ent;
    eptr.assign(tiles + 1, 0);
    {
        std::vector<std::pair<int, int2>> e; // (tile, entry)
        for (int f = 0; f < nfr; f++) {
            const MfFrontDev& d = fr[f];
            const int* first = P.idx.data() + d.idx0;
            const int* last = first + d.npiv + d.nrow;
            for (int l = 0; l < d.npiv; l++) {
                const int k = first[l];
                e.push_back({d.tile0 + mf_tix(d.nt, l / 8, l / 8), make_int2(-k - 1, 9 * (l % 8))});
                for (int pb = col_ptr[k]; pb < col_ptr[k + 1]; pb++) {
                    if (goff_ptr[pb] == goff_ptr[pb + 1]) continue;
                    const int m = (int)(std::lower_bound(first, last, row[pb]) - first), pos = m < d.npiv ? m : 8 * d.P + (m - d.npiv);
                    e.push_back({d.tile0 + mf_tix(d.nt, pos / 8, l / 8), make_int2(pb, 8 * (pos % 8) + l % 8)});
                }
            }
        }
        for (const auto& x : e) eptr[x.first + 1]++;
        for (int64_t t = 0; t < tiles; t++) eptr[t + 1] += eptr[t];
        ent.resize(e.size());
        std::vector<int> fill(eptr.begin(), eptr.end() - 1);
        for (const auto& x : e) ent[fill[x.first]++] = x.second;
    }
    // the tasks: level by level from the leaves, a level's whole fronts first, then its tiles column by column over all
    // its fronts; then the backward solves from the root down, last panels first
    std::vector<int4>& task = Y.task;
    for (int L = 0; L < nlev; L++) {
        int cols = 0;
        const size_t t0 = task.size();
        for (int f = P.level_ptr[L]; f < P.level_ptr[L + 1]; f++) {
            if (alone(f)) task.push_back(make_int4(f, 0, 0, MF_FRONT));
            else cols = std::max(cols, fr[f].nt);
        }
        for (int j = 0; j < cols; j++)
            for (int f = P.level_ptr[L]; f < P.level_ptr[L + 1]; f++) {
                const int end = fr[f].parent >= 0 ? fr[f].nt : fr[f].P; // (a root's Schur complement is nobody's)
                if (alone(f) || j >= end) continue;
                for (int i = j; i < fr[f].nt; i++) task.push_back(make_int4(f, i, j, MF_TILE));
            }
        Y.widest = std::max(Y.widest, (int)(task.size() - t0));
    }
    Y.nfactor = (int)task.size();
    for (int L = nlev - 1; L >= 0; L--) {
        int cols = 0;
        const size_t t0 = task.size();
        for (int f = P.level_ptr[L]; f < P.level_ptr[L + 1]; f++) cols = std::max(cols, fr[f].P);
        for (int b = 0; b < cols; b++)
            for (int f = P.level_ptr[L]; f < P.level_ptr[L + 1]; f++)
                if (b < fr[f].P) task.push_back(make_int4(f, 0, fr[f].P - 1 - b, MF_BACK));
        Y.widest_back = std::max(Y.widest_back, (int)(task.size() - t0));
    }
    return Y;
}

} // namespace blg
