// FP64 ("plain") step kernels.  Compiled with --fmad=false so that every FP64
// operation rounds exactly as written, which makes the step bit-identical to
// the CPU oracle.
#include <algorithm>
#include "step_kernel.cuh"
#include "kernels.h"

namespace godar {

static_assert(sizeof(PairRec64) == FP64_PAIR_REC_BYTES, "pair record size");
static_assert(FS64_COUNT == FP64_FLOE_SUMS, "floe sums");

static int fp64_grid(long long n, int block)
{
    return (int)std::max(1LL, std::min<long long>((n + block - 1) / block, 148LL * (4096 / block)));
}

void launch_pairs_fp64(const Views &V, int cur, int n, const int *plist, const unsigned *erow, unsigned char *pfl,
                       FP64List L, void *rec, int block, cudaStream_t st)
{
    launch_step(V.pdl != 0, k_pairs_fp64, fp64_grid(n, block), block, st, V, cur, n, plist, erow, pfl, L,
                (PairRec64 *)rec);
}

void launch_pairs_list_fp64(const Views &V, int cur, int n, unsigned char *pfl, FP64List L, void *rec, int block,
                            cudaStream_t st)
{
    // the list's length is known on the device only: at most one wave, grid-stride
    const int grid = (int)std::max(1LL, std::min<long long>(((long long)n + block - 1) / block, 148LL * (1024 / block)));
    launch_step(V.pdl != 0, k_pairs_list_fp64<false>, grid, block, st, V, cur, L, pfl, (PairRec64 *)rec);
}

void launch_row_sums_fp64(const Views &V, int cur, int diag, int light, const unsigned char *pfl, const void *rec,
                          const int *lo_n, const int *up_n, double *fs, int block, cudaStream_t st)
{
    const PairRec64 *r = (const PairRec64 *)rec;
    if (diag) launch_step(V.pdl != 0, k_row_sums_fp64<true, false>, fp64_grid(V.N, block), block, st, V, cur, pfl, r, lo_n, up_n, fs);
    else if (light) launch_step(V.pdl != 0, k_row_sums_fp64<false, true>, fp64_grid(V.N, block), block, st, V, cur, pfl, r, lo_n, up_n, fs);
    else launch_step(V.pdl != 0, k_row_sums_fp64<false, false>, fp64_grid(V.N, block), block, st, V, cur, pfl, r, lo_n, up_n, fs);
}

// Plain steps of sheltering batches too large for the merged steps.
void launch_pairs_shel_fp64(const Views &V, int cur, int n, const int *plist, const unsigned *erow,
                            unsigned char *pfl, void *rec, cudaStream_t st)
{
    SmallArgs64 A{};
    A.n = n; A.plist = plist; A.erow = erow; A.pfl = pfl; A.rec = (PairRec64 *)rec;
    if (n > 0) launch_step(V.pdl != 0, k_step_pairs_shel_fp64, SHEL_WAVE / SHEL_THREADS, SHEL_THREADS, st, V, A, cur);
}

// The two kernels of k_pairs_diag_fp64 (the list's length is known on the device
// only: at most one wave, grid-stride).
template <class Launch>
static void pairs_diag(const Views &V, int cur, int E, const unsigned *erow, unsigned char *pfl, FP64List L, void *rec,
                       Launch launch)
{
    launch(k_pairs_diag_fp64, fp64_grid(E, 128), 128, V, cur, E, erow, pfl, L, (PairRec64 *)rec);
    launch(k_pairs_list_fp64<true>, std::min((E + 127) / 128, 148 * 8), 128, V, cur, L, pfl, (PairRec64 *)rec);
}

void launch_pairs_diag_fp64(const Views &V, int cur, int E, int shelter, const unsigned *erow, unsigned char *pfl,
                            FP64List L, void *rec, cudaStream_t st)
{
    if (E <= 0) return;
    if (shelter) {
        SmallArgs64 A{};
        A.n = A.E = E; A.erow = erow; A.pfl = pfl; A.rec = (PairRec64 *)rec;
        launch_step(V.pdl != 0, k_step_pairs_fp64<true, 4>, fp64_grid(E, 128), 128, st, V, A, cur);
        return;
    }
    pairs_diag(V, cur, E, erow, pfl, L, rec, [&](auto kern, int grid, int block, auto... args) {
        launch_step(V.pdl != 0, kern, grid, block, st, args...);
    });
}

void launch_group_sums_fp64(const Views &V, int cur, const unsigned char *pfl, const void *rec, const int *lo_n,
                            const int *up_n, double *fs, cudaStream_t st)
{
    launch_step(V.pdl != 0, k_group_sums_fp64, (V.N + GRP_FLOES - 1) / GRP_FLOES, SMALL_THREADS, st, V, cur, pfl,
                (const PairRec64 *)rec, lo_n, up_n, fs);
}

void launch_floes_fp64(const Views &V, int cur, int diag, int sic, int walls, int light, const double *fs, int *nwork, int block,
                       cudaStream_t st)
{
    const int grid = fp64_grid(V.N, block);
    if (walls) {
        if (diag) launch_step(V.pdl != 0, k_floes_fp64<true, true, false>, grid, block, st, V, cur, sic, fs, nwork);
        else launch_step(V.pdl != 0, k_floes_fp64<false, true, false>, grid, block, st, V, cur, sic, fs, nwork);
    } else {
        if (diag) launch_step(V.pdl != 0, k_floes_fp64<true, false, false>, grid, block, st, V, cur, sic, fs, nwork);
        else if (light) launch_step(V.pdl != 0, k_floes_fp64<false, false, true>, grid, block, st, V, cur, sic, fs, nwork);
        else launch_step(V.pdl != 0, k_floes_fp64<false, false, false>, grid, block, st, V, cur, sic, fs, nwork);
    }
}

int launch_steps_fp64(const Views &V, ClusterLimit &most, int cur, int K, int diag_last, int base, int n, int E, int NB,
                       int shelter, int walls,
                       const int *plist, const unsigned *erow, unsigned char *pfl, void *rec, const int *lo_n,
                       const int *up_n, double *drag, FP64List L, int *out, int *done, cudaStream_t st)
{
    SmallArgs64 A;
    A.cur = cur; A.K = K; A.diag_last = diag_last; A.base = base;
    A.n = n; A.E = E; A.plist = plist; A.erow = erow; A.pfl = pfl; A.rec = (PairRec64 *)rec;
    A.lo_n = lo_n; A.up_n = up_n; A.drag = drag; A.nd = V.N; A.out = out; A.done = done;
    const long long items = (long long)n + V.N;
    int kernels = 0, first = 0;
    if (!shelter && items <= ONE_CLUSTER_FP64) {
        const int blocks = cluster_blocks(items, one_block_fp64(V.N, n, NB));
        auto W = A;
        if (diag_last && diag_apart(V.N, E, blocks, true)) {
            W.K = K - 1;
            W.diag_last = 0;
        }
        if (W.K > 0 && launch_cluster(most, V.pdl != 0, k_steps_fp64, blocks, st, V, W)) {
            kernels = 1;
            first = W.K;
        }
        if (first == K) return kernels;
    }
    const GroupSums how = group_sums(V.N, shelter, n);
    // the drag planes of floes out of sheltering fields, then the sums
    double *fs = drag + 8 * (size_t)V.N;
    const auto launch = [&](auto kern, int grid, int block, auto... args) {
        launch_step(V.pdl != 0, kern, grid, block, st, args...);
        kernels++;
    };
    for (int k = first; k < K; k++) {
        const int c = cur ^ (k & 1);
        const bool diag = diag_last && k == K - 1;
        const long long work = (long long)(diag ? E : n) + 32 + V.N;
        const int gp = fp64_grid(work, 128);
        const bool dense = work > 148 * 2 * 128;
        // (nothing to visit: the update computes its drag itself)
        const bool apart = diag && diag_sums_apart_fp64(V.N, E, NB);
        A.drag = !apart && (diag || n > 0) ? drag : nullptr;
        A.nd = A.drag ? V.N : 0;
        if (apart && !shelter) pairs_diag(V, c, E, erow, pfl, L, rec, launch);
        else if (diag) launch(dense ? k_step_pairs_fp64<true, 4> : k_step_pairs_fp64<true, 2>, gp, 128, V, A, c);
        else if (shelter && n > SHEL_WAVE) launch(k_step_pairs_shel_fp64, SHEL_WAVE / SHEL_THREADS, SHEL_THREADS, V, A, c);
        else if (n > 0) launch(dense ? k_step_pairs_fp64<false, 4> : k_step_pairs_fp64<false, 2>, gp, 128, V, A, c);
        const int groups = (V.N + GRP_FLOES - 1) / GRP_FLOES;
        if (apart) {
            // (every plane of the sums: the drag is the update's)
            const int block = V.N > 148 * 256 ? 128 : 32;      // (on as many SMs as there are blocks for)
            launch(k_row_sums_fp64<true, false>, fp64_grid(V.N, block), block, V, c, (const unsigned char *)pfl,
                   (const PairRec64 *)A.rec, lo_n, up_n, drag);
            launch(walls ? k_step_update_fp64<true, true> : k_step_update_fp64<true, false>, fp64_grid(V.N, 64), 64, V,
                   A, c, k, (const double *)drag, L.n);
        } else if (diag) {
            launch(walls ? k_step_floes_fp64<true, true> : k_step_floes_fp64<true, false>, fp64_grid(V.N, 64), 64, V, A, c, k);
        } else if (how == SUMS_THREAD) {
            launch(walls ? k_step_floes_fp64<false, true> : k_step_floes_fp64<false, false>, fp64_grid(V.N, 64), 64, V, A, c, k);
        } else if (how == SUMS_GROUP) {
            launch(k_step_floes_grp_fp64, groups, SMALL_THREADS, V, A, c, k);
        } else {
            launch(k_group_sums_fp64, groups, SMALL_THREADS, V, c, pfl, A.rec, lo_n, up_n, fs);
            launch(walls ? k_step_update_fp64<false, true> : k_step_update_fp64<false, false>, fp64_grid(V.N, 64), 64, V, A, c, k, (const double *)fs, L.n);
        }
    }
    return kernels;
}

// Owner entries [0, E) at a rebuild (floes on side `side`, at the rebuild
// positions): whether a pair can act on a step without diagnostics before
// the next rebuild.  Until then every floe stays within skin/2 of where it
// is now (a step that takes one farther ends the chunk and a rebuild
// follows) and radii only shrink (ridging), so a pair whose gap exceeds the
// skin cannot touch; a pair without contact, bond or history in a field
// without sheltering changes nothing on such a step (pair_compute resets a
// history that is already zero).  Kept: pairs within reach (with a margin
// far above rounding), bonded pairs, pairs with a history, every pair of a
// sheltering field.  Also the pairs' flags before the first step.
__global__ void k_fp64_mark(Views V, int side, int E, const unsigned *erow, unsigned char *listed, unsigned char *pfl)
{
    const Hist4<double> *H = (const Hist4<double> *)V.hist[0];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x) {
        const int g = (int)erow[e];
        const InstParams &P = V.P[V.inst[g]];
        const int2 en = V.ent_up[e];
        const int t = en.x, p = en.y;
        const double2 h = *(const double2 *)&H[p];
        const bool hist = (__double_as_longlong(h.x) | __double_as_longlong(h.y)) != 0;
        pfl[p] = hist ? PR_HIST : 0;
        bool keep = P.shelter != 0 || V.bidx[p] >= 0 || hist;
        if (!keep) {
            const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
            const double dx = wrap_d(V.x[side][g] - V.x[side][t], P.nx, px);
            const double dy = wrap_d(V.y[side][g] - V.y[side][t], P.ny, py);
            const double dist = sqrt(dx * dx + dy * dy);
            const double reach = (V.r[side][g] + V.r[side][t]) + P.skin;
            keep = !(dist > reach + 1e-6 * (dist + reach) + 1e-3);
        }
        listed[p] = keep ? 1 : 0;
    }
}

// Every floe's rows reordered (stably) so that the pairs kept by
// k_fp64_mark come first: up_n / lo_n of them in the owner / partner row.
// tmp holds E + L entries.
__global__ void k_fp64_partition(Views V, const unsigned char *listed, int *up_n, int *lo_n, int2 *tmp, int E)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < V.N; g += gridDim.x * blockDim.x) {
        for (int side = 0; side < 2; side++) {
            int2 *ent = side ? V.ent_lo : V.ent_up;
            const int *off = side ? V.lo_off : V.up_off;
            int2 *t = tmp + (side ? E : 0);
            const int a0 = off[g], a1 = off[g + 1];
            int m = a0;
            for (int a = a0; a < a1; a++)
                if (listed[ent[a].y]) t[m++] = ent[a];
            (side ? lo_n : up_n)[g] = m - a0;
            for (int a = a0; a < a1; a++)
                if (!listed[ent[a].y]) t[m++] = ent[a];
            for (int a = a0; a < a1; a++) ent[a] = t[a];
        }
    }
}

// The owner-row positions the plain steps' screen visits: the first up_n[g]
// of every row, at pos[g] in the list.
__global__ void k_fp64_list(const int *up_off, const int *up_n, const int *pos, int N, int *plist)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < N; g += gridDim.x * blockDim.x) {
        const int a0 = up_off[g], q = pos[g];
        for (int k = 0; k < up_n[g]; k++) plist[q + k] = a0 + k;
    }
}

// The bonds' working order, by the slot of the lower-id floe: the own bonds of
// every slot, counted; from their scan (wfo) the order itself and the working
// copies.
__global__ void k_fp64_bond_counts(Views V, int side, int *cnt)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < V.N; s += gridDim.x * blockDim.x) {
        const int gl = V.P[V.inst[s]].off + V.id[side][s];
        cnt[s] = V.bond_off[gl + 1] - V.bond_off[gl];
    }
}

__global__ void k_fp64_bond_work(Views V, int side, const int *wfo, int *perm, BondDyn *wdyn, BondGeom64 *wgeo)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < V.N; s += gridDim.x * blockDim.x) {
        const int gl = V.P[V.inst[s]].off + V.id[side][s];
        const int b0 = V.bond_off[gl], b1 = V.bond_off[gl + 1], w0 = wfo[s];
        for (int b = b0; b < b1; b++) {
            const int w = w0 + (b - b0);
            const BondStat c = V.bstat[b];
            BondGeom64 q;
            q.rb = c.rb; q.hb = c.hb; q.lb = c.lb; q.sb = c.sb; q.ib = c.ib;
            perm[w] = b;
            wdyn[w] = V.bdyn[0][b];
            wgeo[w] = q;
        }
    }
}

void launch_fp64_bonds(const Views &V, int side, int *cnt, int *wfo, int *scan_scratch, int *perm, BondDyn *wdyn,
                       BondGeom64 *wgeo, cudaStream_t st)
{
    k_fp64_bond_counts<<<fp64_grid(V.N, 256), 256, 0, st>>>(V, side, cnt);
    scan_excl(cnt, wfo, V.N, scan_scratch, st);
    k_fp64_bond_work<<<fp64_grid(V.N, 128), 128, 0, st>>>(V, side, wfo, perm, wdyn, wgeo);
}

void launch_fp64_rows(const Views &V, int side, int E, const unsigned *erow, unsigned char *pfl,
                      unsigned char *listed, int *up_n, int *lo_n, int2 *tmp, int *pos, int *scan_scratch, int *plist, cudaStream_t st)
{
    if (E > 0) k_fp64_mark<<<fp64_grid(E, 256), 256, 0, st>>>(V, side, E, erow, listed, pfl);
    k_fp64_partition<<<fp64_grid(V.N, 128), 128, 0, st>>>(V, listed, up_n, lo_n, tmp, E);
    scan_excl(up_n, pos, V.N, scan_scratch, st);
    k_fp64_list<<<fp64_grid(V.N, 128), 128, 0, st>>>(V.up_off, up_n, pos, V.N, plist);
}

}  // namespace godar
