// Device-to-host outputs: per-floe fields back in reference index order, and
// the pair lists the reference writes at output steps
// (diagnostics_outputs.f90:157-167, mpi_coms.f90:691-796).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace godar {

// One value of the state (field codes GODAR_F_*, GATHER_DTB1 ..) or of the
// last diagnostic step.
GD_DEV double field_value(const Views &V, int cur, int s, int field)
{
    switch (field) {
    case 0: return V.x[cur][s];
    case 1: return V.y[cur][s];
    case 2: return V.u[cur][s];
    case 3: return V.v[cur][s];
    case 4: return V.r[cur][s];
    case 5: return V.h[cur][s];
    case 6: return V.th[cur][s];
    case 7: return V.om[cur][s];
    // wall histories, for checkpoints
    case GATHER_DTB1: return V.dtb1[cur][s];
    case GATHER_DTB1 + 1: return V.dtb2[cur][s];
    case GATHER_DTB1 + 2: return V.thb1[cur][s];
    case GATHER_DTB1 + 3: return V.thb2[cur][s];
    default: return V.diag[(size_t)(field - 8) * V.N + s];
    }
}

// all = 0: one instance at slots [off, off+n), out in its id order; all = 1:
// every instance, out concatenated by instance (offset P.off) in id order.
__global__ void k_gather_field(Views V, int cur, int off, int n, int field, double *out, int all)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int s = off + k;
        out[(all ? V.P[V.inst[s]].off : 0) + V.id[cur][s]] = field_value(V, cur, s, field);
    }
}

// Several fields of one instance at slots [off, off+n), each in id order:
// field q at out + q n.
__global__ void k_gather_fields(Views V, int cur, int off, int n, FieldList F, double *out)
{
    const int q = blockIdx.y;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        out[(size_t)q * n + V.id[cur][off + k]] = field_value(V, cur, off + k, F.code[q]);
}

// The pair lists.  which: 0 candidates, 1 contacts (pdn of the last
// diagnostic step), 2 live bonds.  A list is in ascending (i, j): the pairs
// are counted by their lower id, the counts scanned, and every row's pairs
// written at their place, ascending in j, so the host has nothing to sort
// (sorting there took most of a read-back: 0.4 ms for 5,300 bonds).  A group
// of lanes takes a row and places its pairs by their rank; a row of more than
// CAP pairs is ranked by its whole block, since a large floe among small ones
// has thousands (one thread inserting 3,272 of them by distance took 100 ms).

// Row item k (0 .. n-1) of the instance at [off, off + n): for lists 0 and 1
// the owner entries of slot off + k, for bonds those of reference id k.
// Returns the lower id.
GD_DEV int list_row(const Views &V, int cur, int off, int which, int k, int &e0, int &e1)
{
    const int *first = which == 2 ? V.bond_off : V.up_off;
    e0 = first[off + k];
    e1 = first[off + k + 1];
    return which == 2 ? k : V.id[cur][off + k];
}

// Whether entry e of a row is in the list, its higher id and value.
GD_DEV bool list_entry(const Views &V, int cur, int which, int e, int &j, double &v)
{
    if (which == 2) {
        const BondDyn d = V.bdyn[cur][e];
        j = V.bond_hi[e];
        v = d.dmg;
        return d.flag == 1;
    }
    const int2 en = V.ent_up[e];
    const float dn = V.pdn[en.y];
    if (dn != dn || (which == 1 && !(dn > 0.0f))) return false;
    j = V.id[cur][en.x];
    v = (double)dn;
    return true;
}

// cnt[lower id]: the pairs of every row.
__global__ void __launch_bounds__(256) k_list_counts(Views V, int cur, int off, int n, int which, int *cnt)
{
    const int sub = threadIdx.x & (GRP - 1), step = gridDim.x * (blockDim.x / GRP);
    // every lane of a warp runs the same rounds
    for (int w = blockIdx.x * (blockDim.x / GRP) + (threadIdx.x & ~31) / GRP; w < n; w += step) {
        const int k = w + (threadIdx.x & 31) / GRP;
        int e0 = 0, e1 = 0, c = 0, id = 0;
        if (k < n) id = list_row(V, cur, off, which, k, e0, e1);
        for (int e = e0 + sub; e < e1; e += GRP) {
            int j;
            double v;
            c += list_entry(V, cur, which, e, j, v);
        }
#pragma unroll
        for (int o = GRP / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (k < n && sub == 0) cnt[id] = c;
    }
}

// The length of the list only (total: zero before).
__global__ void __launch_bounds__(256) k_list_length(Views V, int cur, int off, int n, int which, int *total)
{
    const int sub = threadIdx.x & (GRP - 1), step = gridDim.x * (blockDim.x / GRP);
    int c = 0;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) / GRP; k < n; k += step) {
        int e0, e1;
        list_row(V, cur, off, which, k, e0, e1);
        for (int e = e0 + sub; e < e1; e += GRP) {
            int j;
            double v;
            c += list_entry(V, cur, which, e, j, v);
        }
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(total, c);
}

// Every pair at base[lower id] + its rank in its row, up to cap of them (base:
// n + 1).
constexpr int LIST_THREADS = 128, LIST_CAP = 64;
__global__ void __launch_bounds__(LIST_THREADS) k_list_fill(Views V, int cur, int off, int n, int which,
                                                            const int *base, int cap, int *pi, int *pj, double *val)
{
    constexpr int T = LIST_THREADS;
    __shared__ double bag_v[T / GRP][LIST_CAP];
    __shared__ int bag_j[T / GRP][LIST_CAP];
    __shared__ int tile[T];
    __shared__ int whole[T / GRP];            // rows for the whole block (-1: none)
    const int sub = threadIdx.x & (GRP - 1), grp = threadIdx.x / GRP;
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    const unsigned gmask = ((1u << GRP) - 1u) << (threadIdx.x & 31 & ~(GRP - 1));
    for (int b = blockIdx.x * (T / GRP); b < n; b += gridDim.x * (T / GRP)) {
        int e0 = 0, e1 = 0, id = 0, m = 0, at = 0;
        if (b + grp < n) {
            id = list_row(V, cur, off, which, b + grp, e0, e1);
            at = base[id];
            m = at < cap ? base[id + 1] - at : 0;
        }
        const bool lng = m > LIST_CAP;
        if (lng || m == 0) e1 = e0;
        int c = 0;
        for (int e = e0; __any_sync(0xffffffffu, e < e1); e += GRP) {
            int j = 0;
            double v = 0.0;
            const bool in = e + sub < e1 && list_entry(V, cur, which, e + sub, j, v);
            const unsigned bal = __ballot_sync(0xffffffffu, in) & gmask;
            if (in) {
                const int q = c + __popc(bal & below);
                bag_j[grp][q] = j;
                bag_v[grp][q] = v;
            }
            c += __popc(bal);
        }
        __syncwarp();
        for (int q = sub; q < c; q += GRP) {
            const int j = bag_j[grp][q];
            int r = at;
            for (int k = 0; k < c; k++) r += bag_j[grp][k] < j;
            if (r < cap) {
                pi[r] = id;
                pj[r] = j;
                val[r] = bag_v[grp][q];
            }
        }
        if (sub == 0) whole[grp] = lng ? b + grp : -1;
        if (!__syncthreads_or(lng)) continue;
        for (int g = 0; g < T / GRP; g++) {
            if (whole[g] < 0) continue;
            id = list_row(V, cur, off, which, whole[g], e0, e1);
            at = base[id];
            for (int e = e0; e < e1; e += T) {
                int j = 0, r = at;
                double v = 0.0;
                const bool in = e + (int)threadIdx.x < e1 && list_entry(V, cur, which, e + threadIdx.x, j, v);
                for (int t = e0; t < e1; t += T) {
                    int tj = 0x7fffffff;
                    double tv;
                    if (t + (int)threadIdx.x < e1 && !list_entry(V, cur, which, t + threadIdx.x, tj, tv)) tj = 0x7fffffff;
                    __syncthreads();
                    tile[threadIdx.x] = tj;
                    __syncthreads();
                    if (in) {
                        const int top = min(T, e1 - t);
#pragma unroll 8
                        for (int k = 0; k < top; k++) r += tile[k] < j;
                    }
                }
                if (in && r < cap) {
                    pi[r] = id;
                    pj[r] = j;
                    val[r] = v;
                }
            }
        }
        __syncthreads();          // (the rows' marks are read until here)
    }
}

// The whole list of a small field of short rows by one block, the counts in
// shared memory: one launch instead of three (count, scan, fill).  A thread
// takes a row and inserts up to LIST_SHORT pairs at their place; the block's
// warps rank longer rows.  n floes, entries of all rows: bonds of 1,021 floes
// 57 us a call against 78 by groups of lanes and 73 in three launches, of 4,096
// 81 and 79.  Lists made from the neighbour rows end sooner, at half as many
// floes or more than LIST_ONE_ROW entries a floe (4,096 floes, 23,000
// candidates: 288 us, and 121 in three launches).
constexpr int LIST_ONE_BLOCK = 4096, LIST_ONE_ROW = 8, LIST_SHORT = 16;
__global__ void __launch_bounds__(1024) k_list_pairs(Views V, int cur, int off, int n, int which, int cap, int *pi,
                                                     int *pj, double *val, int *total)
{
    __shared__ int cnt[LIST_ONE_BLOCK + 1];
    __shared__ int sums[32];
    __shared__ int longs[LIST_ONE_BLOCK], nlong;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) nlong = 0;
    for (int k = tid; k < n; k += 1024) {
        int e0, e1, c = 0;
        const int id = list_row(V, cur, off, which, k, e0, e1);
        for (int e = e0; e < e1; e++) {
            int j;
            double v;
            c += list_entry(V, cur, which, e, j, v);
        }
        cnt[id] = c;
    }
    __syncthreads();
    const int per = (n + 1023) / 1024, k0 = min(tid * per, n), k1 = min(k0 + per, n);
    int own = 0;
    for (int k = k0; k < k1; k++) own += cnt[k];
    int pre = own;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += v;
    }
    if (lane == 31) sums[warp] = pre;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; w++) before += sums[w];
    int at = before + pre - own;
    if (tid == 1023) *total = cnt[n] = before + pre;
    for (int k = k0; k < k1; k++) {
        const int c = cnt[k];
        cnt[k] = at;
        at += c;
    }
    __syncthreads();
    if (cap <= 0) return;
    for (int k = tid; k < n; k += 1024) {
        int e0, e1;
        const int id = list_row(V, cur, off, which, k, e0, e1);
        const int a = cnt[id], m = cnt[id + 1] - a;
        if (m == 0 || a >= cap) continue;
        if (m > LIST_SHORT || a + m > cap) {
            longs[atomicAdd(&nlong, 1)] = k;
            continue;
        }
        int top = a;
        for (int e = e0; e < e1; e++) {
            int j;
            double v;
            if (!list_entry(V, cur, which, e, j, v)) continue;
            int q = top++;
            while (q > a && pj[q - 1] > j) {
                pj[q] = pj[q - 1];
                val[q] = val[q - 1];
                q--;
            }
            pi[top - 1] = id;
            pj[q] = j;
            val[q] = v;
        }
    }
    __syncthreads();
    for (int w = warp; w < nlong; w += 32) {
        int e0, e1;
        const int id = list_row(V, cur, off, which, longs[w], e0, e1);
        for (int e = e0; e < e1; e += 32) {
            int j = 0, r = cnt[id];
            double v = 0.0;
            const bool in = e + lane < e1 && list_entry(V, cur, which, e + lane, j, v);
            for (int t = e0; t < e1; t += 32) {
                int tj = 0x7fffffff;
                double tv;
                if (t + lane < e1 && !list_entry(V, cur, which, t + lane, tj, tv)) tj = 0x7fffffff;
#pragma unroll
                for (int q = 0; q < 32; q++) r += __shfl_sync(0xffffffffu, tj, q) < j;
            }
            if (in && r < cap) {
                pi[r] = id;
                pj[r] = j;
                val[r] = v;
            }
        }
    }
}

// Per instance (one block each): total momentum (x, y), kinetic energy of
// translation and rotation, and the largest speed of its floes on side cur
// (mass = rho_ice pi h r^2 and inertia = m r^2 / 2, floe_properties,
// physics.f90:179-198), summed over a block-stride loop and a fixed tree in
// shared memory: deterministic for a given state in a given memory order of
// the floes (their cell order at the last neighbour rebuild).
// It runs beside the next step, whose one-wave kernels wait for the slots its
// blocks hold, so its latency counts: the chains of sums stay those of
// SUM_THREADS threads, but four times as many threads load the floes and form
// the terms (a round ahead of the sums), and each quarter adds one component.
// 512 fields, 2.2 M floes: 60 -> 33 us (one field's block of 256 threads took
// its loads one floe at a time; the largest field, 16,384 floes, is the tail).
constexpr int SUM_THREADS = 256;
constexpr int SUM_U = 1;
__global__ void __launch_bounds__(4 * SUM_THREADS, 2) k_instance_summary(Views V, int cur, double4 *out)
{
    constexpr int T = 4 * SUM_THREADS;
    __shared__ double term[4][SUM_U * T];
    const InstParams &P = V.P[blockIdx.x];
    const int n = P.n, off = P.off;
    const double rp = P.rhoice * P.pi;
    const int part = threadIdx.x / SUM_THREADS, t = threadIdx.x % SUM_THREADS;
    double a = 0.0;
    double r[SUM_U], h[SUM_U], u[SUM_U], v[SUM_U], om[SUM_U];
    auto load = [&](int base) {
#pragma unroll
        for (int q = 0; q < SUM_U; q++) {
            const int i = off + min(base + q * T + (int)threadIdx.x, n - 1);
            r[q] = V.r[cur][i]; h[q] = V.h[cur][i];
            u[q] = V.u[cur][i]; v[q] = V.v[cur][i]; om[q] = V.om[cur][i];
        }
    };
    if (n > 0) load(0);
    for (int base = 0; base < n; base += SUM_U * T) {
#pragma unroll
        for (int q = 0; q < SUM_U; q++) {
            const double m = (rp * h[q]) * (r[q] * r[q]);
            const double in = (0.5 * m) * (r[q] * r[q]);
            const double s2 = u[q] * u[q] + v[q] * v[q];
            const int at = q * T + threadIdx.x;
            term[0][at] = m * u[q];
            term[1][at] = m * v[q];
            term[2][at] = (0.5 * m) * s2 + (0.5 * in) * (om[q] * om[q]);
            term[3][at] = s2;
        }
        if (base + SUM_U * T < n) load(base + SUM_U * T);
        __syncthreads();
        const double *w = term[part] + t;
        const int m = min((n - base - t + SUM_THREADS - 1) / SUM_THREADS, 4 * SUM_U);
        if (part < 3) {
            for (int k = 0; k < m; k++) a = a + w[k * SUM_THREADS];
        } else {
            for (int k = 0; k < m; k++) a = fmax(a, w[k * SUM_THREADS]);
        }
        __syncthreads();
    }
    // (monotone: the root of the largest is the largest root)
    if (part == 3) a = sqrt(a);
    double *red = term[part];
    red[t] = a;
    __syncthreads();
    for (int w = SUM_THREADS / 2; w > 0; w >>= 1) {
        if (t < w) red[t] = part < 3 ? red[t] + red[t + w] : fmax(red[t], red[t + w]);
        __syncthreads();
    }
    if (t == 0) reinterpret_cast<double *>(out + blockIdx.x)[part] = red[0];
}

void launch_instance_summary(const Views &V, int cur, double *out, cudaStream_t st)
{
    if (V.ninst > 0) k_instance_summary<<<V.ninst, 4 * SUM_THREADS, 0, st>>>(V, cur, reinterpret_cast<double4 *>(out));
}

// The four forcing numbers of every field into its parameters, read from
// pinned host memory: one small kernel (a strided copy of 512 rows held the
// stream longer).
__global__ void k_set_forcing(InstParams *P, int ni, const double4 *uvw)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ni) return;
    const double4 f = uvw[k];
    P[k].ua = f.x; P[k].va = f.y; P[k].uw = f.z; P[k].vw = f.w;
}

void launch_set_forcing(InstParams *P, int ni, const double *uvw, cudaStream_t st)
{
    k_set_forcing<<<(ni + 255) / 256, 256, 0, st>>>(P, ni, reinterpret_cast<const double4 *>(uvw));
}

void launch_gather_field(const Views &V, int cur, int inst, int off, int n, int field, double *out, cudaStream_t st)
{
    const int grid = n > 0 ? (n + 255) / 256 : 1;
    k_gather_field<<<grid < 2048 ? grid : 2048, 256, 0, st>>>(V, cur, off, n, field, out, inst < 0 ? 1 : 0);
}

void launch_gather_fields(const Views &V, int cur, int off, int n, const FieldList &F, double *out, cudaStream_t st)
{
    const int grid = n > 0 ? (n + 255) / 256 : 1;
    k_gather_fields<<<dim3(grid < 1024 ? grid : 1024, F.n), 256, 0, st>>>(V, cur, off, n, F, out);
}

const int *launch_list_pairs(const Views &V, int cur, int off, int n, long long entries, int which, int cap, int *pi,
                             int *pj, double *val, int *total, int *cnt, int *base, int *scan_scratch,
                             cudaStream_t st)
{
    if (which == 2 ? n <= LIST_ONE_BLOCK : n <= LIST_ONE_BLOCK / 2 && entries <= (long long)LIST_ONE_ROW * n) {
        k_list_pairs<<<1, 1024, 0, st>>>(V, cur, off, n, which, cap, pi, pj, val, total);
        return total;
    }
    const auto grid = [&](int per) { return (int)std::min<long long>(((long long)n + per - 1) / per, 148 * 16); };
    if (cap <= 0) {
        // (two launches where the counts and their scan are four)
        cudaMemsetAsync(total, 0, sizeof(int), st);
        k_list_length<<<grid(256 / GRP), 256, 0, st>>>(V, cur, off, n, which, total);
        return total;
    }
    k_list_counts<<<grid(256 / GRP), 256, 0, st>>>(V, cur, off, n, which, cnt);
    scan_excl(cnt, base, n, scan_scratch, st);
    k_list_fill<<<grid(LIST_THREADS / GRP), LIST_THREADS, 0, st>>>(V, cur, off, n, which, base, cap, pi, pj, val);
    return base + n;
}

}  // namespace godar

// ------------------------------------------------------------ relayout
// Batch membership changes.  The host describes the new layout by a few
// numbers a field (RelayoutTable); which field a slot or a bond belongs to, and
// where it comes from, is found on the device.
namespace godar {

// The last k in [0, n) with start[k] <= g (start[0] = 0, ascending).
GD_DEV int field_at(const int *start, int n, int g)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Every new slot: its field, where its floe was (repack, -1: admitted now),
// and its state: a resident floe's from the previous layout; of an admitted
// one its id and empty wall histories (the rest is uploaded).
__global__ void k_relayout_floes(Views Vo, int so, Views Vn, int sn, RelayoutTable T, int *inst, int *repack, int n)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const int k = field_at(T.off, T.ni, g), i = g - T.off[k];
        const int o = T.old_off[k] < 0 ? -1 : T.old_off[k] + i;
        inst[g] = k;
        repack[g] = o;
        if (o < 0) {
            Vn.dtb1[sn][g] = 0.0; Vn.dtb2[sn][g] = 0.0; Vn.thb1[sn][g] = 0.0; Vn.thb2[sn][g] = 0.0;
            Vn.id[sn][g] = i;
            continue;
        }
        Vn.x[sn][g] = Vo.x[so][o]; Vn.y[sn][g] = Vo.y[so][o]; Vn.th[sn][g] = Vo.th[so][o];
        Vn.u[sn][g] = Vo.u[so][o]; Vn.v[sn][g] = Vo.v[so][o]; Vn.om[sn][g] = Vo.om[so][o];
        Vn.r[sn][g] = Vo.r[so][o]; Vn.h[sn][g] = Vo.h[so][o];
        Vn.dtb1[sn][g] = Vo.dtb1[so][o]; Vn.dtb2[sn][g] = Vo.dtb2[so][o];
        Vn.thb1[sn][g] = Vo.thb1[so][o]; Vn.thb2[sn][g] = Vo.thb2[so][o];
        Vn.id[sn][g] = Vo.id[so][o];
    }
}

// bond_off of resident floes, rebased (the floe with reference id k of field b
// keeps its bonds), and the resident bonds moved.
__global__ void k_relayout_bond_off(const int *old_bond_off, int *new_bond_off, const int *inst, RelayoutTable T,
                                    int n)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const int b = inst[g];
        if (T.old_off[b] < 0) continue;
        new_bond_off[g] = old_bond_off[T.old_off[b] + (g - T.off[b])] - T.old_boff[b] + T.boff[b];
    }
}

__global__ void k_relayout_bonds(const int *old_hi, const BondStat *old_st, const BondDyn *old_dy, int *new_hi,
                                 BondStat *new_st, BondDyn *new_dy, RelayoutTable T, int nb)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nb; q += gridDim.x * blockDim.x) {
        const int k = field_at(T.boff, T.ni, q);
        if (T.old_boff[k] < 0) continue;
        const int o = T.old_boff[k] + (q - T.boff[k]);
        new_hi[q] = old_hi[o];
        new_st[q] = old_st[o];
        new_dy[q] = old_dy[o];
    }
}

static int rl_grid(int n) { return n > 0 ? ((n + 255) / 256 < 2368 ? (n + 255) / 256 : 2368) : 1; }

void launch_relayout_floes(const Views &Vo, int so, const Views &Vn, int sn, const RelayoutTable &T, int *inst,
                           int *repack, int n, cudaStream_t st)
{
    k_relayout_floes<<<rl_grid(n), 256, 0, st>>>(Vo, so, Vn, sn, T, inst, repack, n);
}

void launch_relayout_bonds(const int *old_bond_off, int *new_bond_off, const int *inst, const int *old_hi,
                           const BondStat *old_st, const BondDyn *old_dy, int *new_hi, BondStat *new_st,
                           BondDyn *new_dy, const RelayoutTable &T, int n, int nb, cudaStream_t st)
{
    k_relayout_bond_off<<<rl_grid(n), 256, 0, st>>>(old_bond_off, new_bond_off, inst, T, n);
    if (nb > 0) k_relayout_bonds<<<rl_grid(nb), 256, 0, st>>>(old_hi, old_st, old_dy, new_hi, new_st, new_dy, T, nb);
}

__global__ void k_set_int(int *p, int v) { *p = v; }

// Sets one device int in stream order (the value is the launch's argument,
// so no host buffer has to outlive the call).
void launch_set_int(int *p, int v, cudaStream_t st)
{
    k_set_int<<<1, 1, 0, st>>>(p, v);
}

__global__ void k_chunk_end(const int *status, int *hs, int *base, int next)
{
    hs[0] = status[0];
    hs[1] = status[1];
    *base = next;
}

void launch_chunk_end(const int *status, int *hs, int *base, int next, cudaStream_t st)
{
    k_chunk_end<<<1, 1, 0, st>>>(status, hs, base, next);
}

}  // namespace godar
