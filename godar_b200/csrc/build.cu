// Kernel (a): the neighbour search that replaces coretran's kd-tree
// (KdTree build, kdtree_utils.f90:21-24; radius query kNearest,
// stepper.f90:77-78).
//
// One rebuild (all instances of a batch at once):
//   1. k_cell_count, scan, k_cell_scatter: the cell list, by counting (the
//      cell of a floe: its instance's first cell + row-major cell)
//   2. k_cell_place: the floes' state gathered into cell order on the other
//      ping-pong side, floes of one cell in their previous order
//   3. k_nbr_count, scan, k_nbr_fill: the symmetric neighbour superset, every
//      t with dist(s,t) <= r_lo + rtree + skin, lo = the floe of lower id, as
//      owner rows (partners of higher id, by distance; by id in the mixed path)
//      and partner rows (partners of lower id, by id)
//   4. k_row_finish: the pair index of every partner entry (the entry of the
//      lower-id floe's owner row that points back), contact histories from
//      the previous rows by reference ids, bond indices, and what else a
//      fresh row holds
// The step kernel filters the superset with the exact candidate predicate
// every step, so the candidate set is the kd-tree's radius query exactly as
// long as no floe moved more than skin/2 since the rebuild (checked every
// step).  This file is compiled with --fmad=false: distances must round
// exactly as in the step kernel and the CPU oracle.
//
// What bounds it: on small fields the chains of dependent loads of one thread
// per floe (cells, floes, rows) and the number of launches; on large ones the
// same chains at partial occupancy.  So a group of eight lanes takes a floe,
// reads each stencil row as one range, and ranks a row's entries by counting
// instead of inserting them one by one; and the list is built by counting
// (6 launches where the radix sort took 11-16).
#include <algorithm>

#include "cells.cuh"
#include "kernels.h"

namespace godar {

// ------------------------------------------------------------ radix sort
// Tile of RS_THREADS x RS_ITEMS keys per block; item k of the tile is key
// tile_base + round*RS_THREADS + tid, so ranking round by round, warp by warp
// and lane by lane keeps equal digits in input order (stable).
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const uint32_t *keys, int n, int shift, int *counts, int ntiles)
{
    __shared__ int hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        const int i = base + k * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&hist[(keys[i] >> shift) & 255], 1);
    }
    __syncthreads();
    counts[threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(const uint32_t *keys, const int *vals, uint32_t *okeys,
                                                            int *ovals, int n, int shift, const int *offsets, int ntiles)
{
    __shared__ int wcnt[RS_WARPS][256];
    __shared__ int run[256];
    __shared__ int tot[256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    run[tid] = offsets[tid * ntiles + blockIdx.x];
    const int base = blockIdx.x * RS_TILE;
    for (int k = 0; k < RS_ITEMS; k++) {
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) wcnt[w][tid] = 0;
        __syncthreads();
        const int i = base + k * RS_THREADS + tid;
        const bool valid = i < n;
        uint32_t key = 0;
        int val = 0, d = 0;
        if (valid) {
            key = keys[i];
            val = vals[i];
            d = (key >> shift) & 255;
        }
        const unsigned act = __ballot_sync(0xffffffffu, valid);
        unsigned peers = 0;
        int rank = 0;
        if (valid) {
            peers = __match_any_sync(act, d);
            rank = __popc(peers & ((1u << lane) - 1u));
            if (rank == 0) wcnt[warp][d] = __popc(peers);
        }
        __syncthreads();
        {   // exclusive prefix over warps for digit tid
            int acc = 0;
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) {
                const int c = wcnt[w][tid];
                wcnt[w][tid] = acc;
                acc += c;
            }
            tot[tid] = acc;
        }
        __syncthreads();
        if (valid) {
            const int pos = run[d] + wcnt[warp][d] + rank;
            okeys[pos] = key;
            ovals[pos] = val;
        }
        __syncthreads();
        run[tid] += tot[tid];
        __syncthreads();
    }
}

// ------------------------------------------------------------ exclusive scan
// out[i] = sum_{k<i} in[i]; out[n] = total.  Three phases: per-block scan,
// scan of block sums by one block, add.  n may be any int: a batch of sparse
// fields has up to 2^31 - 1 cells, so an index past the end is not an int.
constexpr int SC_THREADS = 512;
constexpr int SC_ITEMS = 4;
constexpr int SC_TILE = SC_THREADS * SC_ITEMS;

GD_DEV int block_excl_scan(int v, int *sh, int &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        int s = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) sh[lane] = s;
    }
    __syncthreads();
    total = sh[(blockDim.x >> 5) - 1];
    const int pre = warp > 0 ? sh[warp - 1] : 0;
    __syncthreads();
    return pre + x - v;
}

__global__ void __launch_bounds__(SC_THREADS) k_scan_tiles(const int *in, int *out, int n, int *tile_sums)
{
    __shared__ int sh[32];
    const int base = blockIdx.x * SC_TILE + threadIdx.x * SC_ITEMS;
    int v[SC_ITEMS], s = 0;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; k++) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    int total;
    int pre = block_excl_scan(s, sh, total);
#pragma unroll
    for (int k = 0; k < SC_ITEMS; k++) {
        if (base + k < n) out[base + k] = pre;
        pre += v[k];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_sums(int *tile_sums, int ntiles, int *total_out)
{
    __shared__ int sh[32];
    int carry = 0;
    for (int base = 0; base < ntiles; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < ntiles ? tile_sums[i] : 0;
        int total;
        const int pre = block_excl_scan(v, sh, total);
        if (i < ntiles) tile_sums[i] = carry + pre;
        carry += total;
    }
    if (threadIdx.x == 0) *total_out = carry;
}

__global__ void k_scan_add(int *out, int n, const int *tile_sums, const int *total, int *out_n)
{
    // (an element a thread)
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < (unsigned)n) out[i] += tile_sums[i / SC_TILE];
    if (blockIdx.x == 0 && threadIdx.x == 0 && out_n) *out_n = *total;
}

// The whole scan by one block: a short one is three launches' latency
// otherwise (a rebuild of a few hundred floes has five of them).
constexpr int SC_SHORT = 8192;
__global__ void __launch_bounds__(1024) k_scan_short(const int *in, int *out, int n)
{
    __shared__ int sh[32];
    constexpr int PER = SC_SHORT / 1024;
    const int base = threadIdx.x * PER;
    int v[PER], s = 0;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    int total;
    int pre = block_excl_scan(s, sh, total);
#pragma unroll
    for (int k = 0; k < PER; k++) {
        if (base + k < n) out[base + k] = pre;
        pre += v[k];
    }
    if (threadIdx.x == 0) out[n] = total;
}

void scan_excl(const int *in, int *out, int n, int *scratch, cudaStream_t st)
{
    // scratch: ntiles + 1 ints; out must hold n + 1 ints
    if (n <= SC_SHORT) {
        k_scan_short<<<1, 1024, 0, st>>>(in, out, n);
        return;
    }
    const int ntiles = (int)(((long long)n + SC_TILE - 1) / SC_TILE);
    k_scan_tiles<<<ntiles, SC_THREADS, 0, st>>>(in, out, n, scratch + 1);
    k_scan_sums<<<1, 1024, 0, st>>>(scratch + 1, ntiles, scratch);
    k_scan_add<<<(int)(((long long)n + 255) / 256), 256, 0, st>>>(out, n, scratch + 1, scratch, out + n);
}

void radix_sort(uint32_t *keys, int *vals, uint32_t *keys_alt, int *vals_alt, int n, int bits,
                int *counts, int *scratch, cudaStream_t st)
{
    const int ntiles = (n + RS_TILE - 1) / RS_TILE;
    const int passes = (bits + 7) / 8;
    uint32_t *ki = keys, *ko = keys_alt;
    int *vi = vals, *vo = vals_alt;
    for (int p = 0; p < passes; p++) {
        const int shift = 8 * p;
        k_radix_hist<<<ntiles, RS_THREADS, 0, st>>>(ki, n, shift, counts, ntiles);
        scan_excl(counts, counts, 256 * ntiles, scratch, st);
        k_radix_scatter<<<ntiles, RS_THREADS, 0, st>>>(ki, vi, ko, vo, n, shift, counts, ntiles);
        uint32_t *tk = ki; ki = ko; ko = tk;
        int *tv = vi; vi = vo; vo = tv;
    }
    if (ki != keys) {
        cudaMemcpyAsync(keys, ki, (size_t)n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
        cudaMemcpyAsync(vals, vi, (size_t)n * sizeof(int), cudaMemcpyDeviceToDevice, st);
    }
}

// ------------------------------------------------------------ cell list
// Floes [s0, s0 + n): their cells and how many each cell has (cnt, zero
// before); after the scan, the cells' floes in any order (cnt back to zero).
__global__ void k_cell_count(Views V, int cur, int s0, int n, uint32_t *keys, int *cnt)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int s = s0 + k;
        const uint32_t c = cell_key(V.P[V.inst[s]], V.x[cur][s], V.y[cur][s]);
        keys[k] = c;
        atomicAdd(&cnt[c], 1);
    }
}

__global__ void k_cell_scatter(int s0, int n, const uint32_t *keys, const int *coff, int *cnt, int *list)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t c = keys[k];
        list[coff[c] + atomicSub(&cnt[c], 1) - 1] = s0 + k;
    }
}

// The floes in cell order, those of a cell in ascending previous slot (a
// floe's place: how many of its cell's floes come before it); old_slot: the
// floe's slot in the previous layout (repack maps pre-sort slots to it; -1 for
// floes new to the batch).
__global__ void k_cell_place(Views V, int cur, const uint32_t *keys, const int *coff, const int *list,
                             const int *repack, int *old_slot)
{
    const int nxt = cur ^ 1;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < V.N; q += gridDim.x * blockDim.x) {
        const int o = list[q];
        const uint32_t c = keys[o];
        const int a = coff[c], b = coff[c + 1];
        int s = a;
        for (int k = a; k < b; k++) s += list[k] < o;
        const double x = V.x[cur][o], y = V.y[cur][o];
        V.x[nxt][s] = x;
        V.y[nxt][s] = y;
        V.th[nxt][s] = V.th[cur][o];
        V.u[nxt][s] = V.u[cur][o];
        V.v[nxt][s] = V.v[cur][o];
        V.om[nxt][s] = V.om[cur][o];
        V.r[nxt][s] = V.r[cur][o];
        V.h[nxt][s] = V.h[cur][o];
        V.dtb1[nxt][s] = V.dtb1[cur][o];
        V.dtb2[nxt][s] = V.dtb2[cur][o];
        V.thb1[nxt][s] = V.thb1[cur][o];
        V.thb2[nxt][s] = V.thb2[cur][o];
        V.id[nxt][s] = V.id[cur][o];
        V.x0[nxt][s] = x;
        V.y0[nxt][s] = y;
        old_slot[s] = repack ? repack[o] : o;
    }
}

// ------------------------------------------------------------ neighbour rows
// Floe s against every floe of the stencil around it that falls to this lane:
// f(t, dist, id of t) when t != s and dist <= r_lo + rtree + skin.
template <class F>
GD_DEV void for_superset(const Views &V, int side, const int *coff, int s, int sub, F f)
{
    const InstParams &P = V.P[V.inst[s]];
    const double xs = V.x[side][s], ys = V.y[side][s], rs = V.r[side][s];
    const int ids = V.id[side][s];
    const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
    walk_cells(P, xs, ys, coff, sub, [&](int t) {
        if (t == s) return;
        const double dx = wrap_d(xs - V.x[side][t], P.nx, px);
        const double dy = wrap_d(ys - V.y[side][t], P.ny, py);
        const double d = sqrt(dx * dx + dy * dy);
        const int idt = V.id[side][t];
        const double rlo = ids < idt ? rs : V.r[side][t];
        if (d <= (rlo + P.rtree) + P.skin) f(t, d, idt);
    });
}

// cnt[s], cnt[N + s]: the partners of lower and of higher id of every floe.
__global__ void __launch_bounds__(256) k_nbr_count(Views V, int side, const int *coff, int *cnt)
{
    const int sub = threadIdx.x & (GRP - 1);
    const int groups = gridDim.x * (blockDim.x / GRP);
    // every lane of a warp runs the same rounds (the sums are warp-wide)
    for (int s0 = blockIdx.x * (blockDim.x / GRP) + (threadIdx.x & ~31) / GRP; s0 < V.N; s0 += groups) {
        const int s = s0 + (threadIdx.x & 31) / GRP;
        int lo = 0, up = 0;
        if (s < V.N) {
            const int ids = V.id[side][s];
            for_superset(V, side, coff, s, sub, [&](int, double, int idt) { if (idt < ids) lo++; else up++; });
        }
#pragma unroll
        for (int o = GRP / 2; o > 0; o >>= 1) {
            lo += __shfl_xor_sync(0xffffffffu, lo, o);
            up += __shfl_xor_sync(0xffffffffu, up, o);
        }
        if (s < V.N && sub == 0) {
            cnt[s] = lo;
            cnt[V.N + s] = up;
        }
    }
}

// Whether entry (da, ida) comes before (db, idb) in a row: partner rows and,
// with up_by_id, owner rows by id; owner rows else by (distance, id).
// up_by_id: the mixed path, whose per-floe sums follow the row order: the
// order then depends only on the reference ids, not on when the rows were
// built (the FP64 path re-sorts its owner rows by distance every step, the
// kd-tree's order).
GD_DEV bool row_before(double da, int ida, double db, int idb, bool by_dist)
{
    return by_dist ? da < db || (da == db && ida < idb) : ida < idb;
}

// An entry of a row longer than a group keeps, before it is ranked.
struct __align__(16) RowEntry {
    double d;
    int t, id;
};

static_assert(sizeof(RowEntry) <= sizeof(Hist4<float>), "raw owner rows lie where the histories go");

// The rows of every floe: off2 is the scan of k_nbr_count's counts (partner
// rows from off2[s], owner rows from off2[N + s] - off2[N]).  A group collects
// its floe's entries in shared memory and places each by its rank.  The rows of
// a floe with more than ROW_CAP partners are collected in global memory (lo_raw,
// up_raw) and ranked by the whole block, a tile of entries in shared memory at
// a time: one lane inserting the 3,272 entries of a large floe among small ones
// took 480 ms, the block 3.
constexpr int ROW_THREADS = 128, ROW_CAP = 112;
__global__ void __launch_bounds__(ROW_THREADS) k_nbr_fill(Views V, int side, const int *coff, const int *off2,
                                                          int up_by_id, int *lo_off, int *up_off, int2 *ent_lo,
                                                          int2 *ent_up, int2 *lo_raw, RowEntry *up_raw,
                                                          int *row_max)
{
    constexpr int T = ROW_THREADS;
    __shared__ GroupBag<ROW_CAP> bags[T / GRP];
    __shared__ int whole[T / GRP];                // floes for the whole block (-1: none)
    __shared__ double tile_d[T];
    __shared__ int tile_id[T];
    const int sub = threadIdx.x & (GRP - 1), grp = threadIdx.x / GRP;
    GroupBag<ROW_CAP> &B = bags[grp];
    const int N = V.N, P = off2[N];
    for (int b = blockIdx.x * (T / GRP); b < N; b += gridDim.x * (T / GRP)) {
        const int s = b + grp;
        if (sub == 0) B.n[0] = B.n[1] = 0;
        __syncwarp();
        const bool on = s < N;
        const int ids = on ? V.id[side][s] : 0;
        const int lo = on ? off2[s] : 0, up = on ? off2[N + s] - P : 0;
        const int m = on ? off2[s + 1] - lo + (off2[N + s + 1] - P) - up : 0;
        const bool lng = m > ROW_CAP;
        if (m > LONG_ROW && sub == 0) atomicMax(row_max, m);
        if (on && sub == 0) {
            lo_off[s] = lo;
            up_off[s] = up;
            if (s == N - 1) {
                lo_off[N] = P;
                up_off[N] = P;
            }
        }
        if (on && !lng) {
            for_superset(V, side, coff, s, sub, [&](int t, double d, int idt) {
                const int k = atomicAdd(&B.n[0], 1);
                B.t[k] = t;
                B.id[k] = idt;
                B.d[k] = d;
            });
        } else if (on) {
            for_superset(V, side, coff, s, sub, [&](int t, double d, int idt) {
                const int u = idt > ids, k = atomicAdd(&B.n[u], 1);
                if (u) {
                    RowEntry e;
                    e.d = d; e.t = t; e.id = idt;
                    up_raw[up + k] = e;
                } else {
                    lo_raw[lo + k] = make_int2(t, idt);
                }
            });
        }
        __syncwarp();
        if (on && !lng) {
            for (int k = sub; k < m; k += GRP) {
                const int idk = B.id[k];
                const double dk = B.d[k];
                const bool u = idk > ids;
                int at = 0;
                for (int j = 0; j < m; j++)
                    at += (B.id[j] > ids) == u && row_before(B.d[j], B.id[j], dk, idk, u && !up_by_id);
                if (u) ent_up[up + at] = make_int2(B.t[k], up + at);      // the pair's index: its own place
                else ent_lo[lo + at] = make_int2(B.t[k], -1);
            }
        }
        if (sub == 0) whole[grp] = lng ? s : -1;
        if (!__syncthreads_or(lng)) continue;
        for (int g = 0; g < T / GRP; g++) {
            if (whole[g] < 0) continue;
            const int lo_g = off2[whole[g]], up_g = off2[N + whole[g]] - P;
            for (int u = 0; u < 2; u++) {
                const int n = bags[g].n[u];
                for (int c = 0; c < n; c += T) {
                    const bool in = c + (int)threadIdx.x < n;
                    RowEntry own;
                    own.d = 0.0; own.t = own.id = 0;
                    if (in && u) {
                        own = up_raw[up_g + c + threadIdx.x];
                    } else if (in) {
                        const int2 e = lo_raw[lo_g + c + threadIdx.x];
                        own.t = e.x; own.id = e.y;
                    }
                    int at = 0;
                    for (int t0 = 0; t0 < n; t0 += T) {
                        const int k = t0 + threadIdx.x;
                        __syncthreads();
                        if (k < n) {
                            tile_d[threadIdx.x] = u ? up_raw[up_g + k].d : 0.0;
                            tile_id[threadIdx.x] = u ? up_raw[up_g + k].id : lo_raw[lo_g + k].y;
                        }
                        __syncthreads();
                        const int top = min(T, n - t0);
#pragma unroll 4
                        for (int j = 0; j < top; j++)
                            at += row_before(tile_d[j], tile_id[j], own.d, own.id, u && !up_by_id);
                    }
                    if (in && u) ent_up[up_g + at] = make_int2(own.t, up_g + at);
                    else if (in) ent_lo[lo_g + at] = make_int2(own.t, -1);
                }
            }
        }
        __syncthreads();          // (the bags and marks are read until here)
    }
}

// What the fresh rows hold besides the partners; a group per floe.
// Partner entries: the pair's index (ST_ROW_OVERFLOW if the partner's owner
// row does not point back) and, mixed, its inverse and no record flag.  Owner
// entries: row, bond index (bonds are sorted by the partner's id; in the FP64
// path counted in the working order, from wfo[s]), no overlap,
// and the contact history by reference ids from the previous rows (old_up_off
// null: zero); mixed, the history flag.
template <typename H4, bool MIXED>
__global__ void __launch_bounds__(256) k_row_finish(Views V, int side, const int *old_slot, const int *old_up_off,
                                                    const int2 *old_ent_up, const int *old_id, const H4 *old_hist,
                                                    const int *up_off, const int *lo_off, const int2 *ent_up,
                                                    int2 *ent_lo, H4 *hist, int *bidx, unsigned *erow, float *pdn,
                                                    unsigned char *pfl, unsigned char *lfl, int *lo_of, const int *wfo)
{
    const int sub = threadIdx.x & (GRP - 1);
    const int groups = gridDim.x * (blockDim.x / GRP);
    for (int s = blockIdx.x * (blockDim.x / GRP) + threadIdx.x / GRP; s < V.N; s += groups) {
        const int ids = V.id[side][s];
        for (int e = lo_off[s] + sub; e < lo_off[s + 1]; e += GRP) {
            const int t = ent_lo[e].x;
            int found = -1;
            for (int q = up_off[t]; q < up_off[t + 1]; q++)
                if (ent_up[q].x == s) { found = q; break; }
            ent_lo[e].y = found;
            if (found < 0) atomicOr(V.status, ST_ROW_OVERFLOW);
            if (MIXED) {
                if (found >= 0) lo_of[found] = e;
                lfl[e] = 0;
            }
        }
        const int e0 = up_off[s], e1 = up_off[s + 1];
        if (e0 == e1) continue;
        const InstParams &P = V.P[V.inst[s]];
        const int os = old_slot[s];
        const int q0 = os >= 0 && old_up_off ? old_up_off[os] : 0, q1 = os >= 0 && old_up_off ? old_up_off[os + 1] : 0;
        const int gl = P.off + ids;
        const int b0 = V.bond_off[gl], b1 = V.bond_off[gl + 1];
        for (int e = e0 + sub; e < e1; e += GRP) {
            const int idt = V.id[side][ent_up[e].x];
            H4 h;
            h.deltat = 0; h.thetarelc = 0; h.fcn = 0; h.fct = 0;
            for (int q = q0; q < q1; q++) {
                const int2 oe = old_ent_up[q];
                if (old_id[oe.x] == idt) { h = old_hist[oe.y]; break; }
            }
            hist[e] = h;
            int lo = b0, hi = b1 - 1, bi = -1;
            while (lo <= hi) {
                const int mid = (lo + hi) >> 1;
                const int v = V.bond_hi[mid];
                if (v == idt) { bi = mid; break; }
                if (v < idt) lo = mid + 1; else hi = mid - 1;
            }
            bidx[e] = !MIXED && bi >= 0 ? wfo[s] + (bi - b0) : bi;
            erow[e] = (unsigned)s;
            pdn[e] = __int_as_float(-1);       // a NaN: not a candidate
            if (MIXED) pfl[e] = h.deltat != 0 || h.thetarelc != 0 ? 1 : 0;     // PF_HIST
        }
    }
}

// Ids, rebuild positions and shapes on both sides (after the histories moved:
// they are found by the previous layout's ids); a batch whose shapes cannot
// change does not write them again.
__global__ void k_copy_ids(Views V, int from)
{
    const int to = from ^ 1;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < V.N; s += gridDim.x * blockDim.x) {
        V.id[to][s] = V.id[from][s];
        V.x0[to][s] = V.x0[from][s];
        V.y0[to][s] = V.y0[from][s];
        V.r[to][s] = V.r[from][s];
        V.h[to][s] = V.h[from][s];
    }
}

// The state fresh rows start from: no error and no expiry, an empty work
// list (nwork's first two; the third is the next rebuild's longest row) and, mixed, no displacement (the contact list holds the gaps at the
// rebuild).
__global__ void k_rows_ready(int *status, int *nwork, unsigned *dsp)
{
    if (threadIdx.x == 0) {
        status[0] = 0;
        status[1] = 0x7fffffff;
    }
    if (threadIdx.x < 3) nwork[threadIdx.x] = 0;
    if (threadIdx.x < 4) dsp[threadIdx.x] = 0;
}

// ------------------------------------------------------------ host side
static int grid_for(long long n, int block)
{
    return n <= 0 ? 1 : (int)std::min<long long>((n + block - 1) / block, 148LL * 16);
}

void launch_cell_list(const Views &V, int cur, int s0, int n, long long C, uint32_t *keys, int *cnt, int *coff,
                      int *list, int *scan_scratch, cudaStream_t st)
{
    cudaMemsetAsync(cnt, 0, (size_t)C * 4, st);
    k_cell_count<<<grid_for(n, 256), 256, 0, st>>>(V, cur, s0, n, keys, cnt);
    scan_excl(cnt, coff, (int)C, scan_scratch, st);
    k_cell_scatter<<<grid_for(n, 256), 256, 0, st>>>(s0, n, keys, coff, cnt, list);
}

void launch_cell_place(const Views &V, int cur, const uint32_t *keys, const int *coff, const int *list,
                       const int *repack, int *old_slot, cudaStream_t st)
{
    k_cell_place<<<grid_for(V.N, 256), 256, 0, st>>>(V, cur, keys, coff, list, repack, old_slot);
}

void launch_nbr_count(const Views &V, int side, const int *coff, int *cnt, int *off2, int *scan_scratch,
                      cudaStream_t st)
{
    k_nbr_count<<<grid_for((long long)V.N * GRP, 256), 256, 0, st>>>(V, side, coff, cnt);
    scan_excl(cnt, off2, 2 * V.N, scan_scratch, st);
}

void launch_nbr_fill(const Views &V, int side, const int *coff, const int *off2, int up_by_id, int *lo_off,
                     int *up_off, int2 *ent_lo, int2 *ent_up, void *lo_raw, void *up_raw, int *row_max,
                     cudaStream_t st)
{
    k_nbr_fill<<<grid_for((long long)V.N * GRP, ROW_THREADS), ROW_THREADS, 0, st>>>(
        V, side, coff, off2, up_by_id, lo_off, up_off, ent_lo, ent_up, (int2 *)lo_raw, (RowEntry *)up_raw, row_max);
}

void launch_row_finish(const Views &V, int mixed, int side, const int *old_slot, const int *old_up_off,
                       const int2 *old_ent_up, const int *old_id, const void *old_hist, const int *up_off,
                       const int *lo_off, const int2 *ent_up, int2 *ent_lo, void *hist, int *bidx, unsigned *erow,
                       float *pdn, unsigned char *pfl, unsigned char *lfl, int *lo_of, const int *wfo,
                       cudaStream_t st)
{
    const int grid = grid_for((long long)V.N * GRP, 256);
    if (mixed)
        k_row_finish<Hist4<float>, true><<<grid, 256, 0, st>>>(
            V, side, old_slot, old_up_off, old_ent_up, old_id, (const Hist4<float> *)old_hist, up_off, lo_off, ent_up,
            ent_lo, (Hist4<float> *)hist, bidx, erow, pdn, pfl, lfl, lo_of, wfo);
    else
        k_row_finish<Hist4<double>, false><<<grid, 256, 0, st>>>(
            V, side, old_slot, old_up_off, old_ent_up, old_id, (const Hist4<double> *)old_hist, up_off, lo_off, ent_up,
            ent_lo, (Hist4<double> *)hist, bidx, erow, pdn, pfl, lfl, lo_of, wfo);
    k_copy_ids<<<grid_for(V.N, 256), 256, 0, st>>>(V, side);
}

void launch_rows_ready(int *status, int *nwork, unsigned *dsp, cudaStream_t st)
{
    k_rows_ready<<<1, 32, 0, st>>>(status, nwork, dsp);
}

}  // namespace godar
