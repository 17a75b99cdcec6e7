// Device-to-host outputs: per-floe fields back in reference index order, and
// the pair lists the reference writes at output steps
// (diagnostics_outputs.f90:157-167, mpi_coms.f90:691-796).
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
// are counted by their lower id, the counts scanned, and every floe writes its
// own pairs at its place, ascending in j, so the host has nothing to sort
// (sorting there took most of a read-back: 0.4 ms for 5,300 bonds).

// The pairs of row item k (0 .. n-1) of the instance at [off, off + n): for
// lists 0 and 1 those of slot off + k, for bonds those of reference id k.
// Calls f(j, value); returns the lower id.
template <class F>
GD_DEV int row_pairs(const Views &V, int cur, int off, int which, int k, F f)
{
    if (which == 2) {
        for (int b = V.bond_off[off + k]; b < V.bond_off[off + k + 1]; b++) {
            const BondDyn d = V.bdyn[cur][b];
            if (d.flag == 1) f(V.bond_hi[b], d.dmg);
        }
        return k;
    }
    const int s = off + k;
    for (int e = V.up_off[s]; e < V.up_off[s + 1]; e++) {
        const int2 en = V.ent_up[e];
        const float dn = V.pdn[en.y];
        if (dn != dn || (which == 1 && !(dn > 0.0f))) continue;
        f(V.id[cur][en.x], (double)dn);
    }
    return V.id[cur][s];
}

GD_DEV int count_row(const Views &V, int cur, int off, int which, int k, int &id)
{
    int c = 0;
    id = row_pairs(V, cur, off, which, k, [&](int, double) { c++; });
    return c;
}

// Row item k's pairs at their place: base[id], each inserted in ascending j
// among those already there.
GD_DEV void write_row(const Views &V, int cur, int off, int which, int k, const int *base, int cap, int *pi, int *pj,
                      double *val)
{
    const int i = which == 2 ? k : V.id[cur][off + k];
    const int a = base[i];
    int m = a;
    row_pairs(V, cur, off, which, k, [&](int j, double v) {
        if (m < cap) {
            int q = m;
            while (q > a && pj[q - 1] > j) {
                pj[q] = pj[q - 1];
                val[q] = val[q - 1];
                q--;
            }
            pi[m] = i;
            pj[q] = j;
            val[q] = v;
        } else {
            // past the caller's capacity: the largest j of this row leaves
            int q = cap;
            while (q > a && pj[q - 1] > j) {
                if (q < cap) { pj[q] = pj[q - 1]; val[q] = val[q - 1]; }
                q--;
            }
            if (q < cap) { pj[q] = j; val[q] = v; }
        }
        m++;
    });
}

__global__ void k_list_counts(Views V, int cur, int off, int n, int which, int *cnt)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        int id;
        const int c = count_row(V, cur, off, which, k, id);
        cnt[id] = c;
    }
}

__global__ void k_list_fill(Views V, int cur, int off, int n, int which, const int *base, int cap, int *pi, int *pj,
                            double *val)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        write_row(V, cur, off, which, k, base, cap, pi, pj, val);
}

// The whole list of a field of up to LIST_ONE_BLOCK floes by one block, the
// counts in shared memory: one launch instead of six (count, three of the
// scan, fill), which is what a list of a few thousand pairs costs.
constexpr int LIST_ONE_BLOCK = 8192;
__global__ void __launch_bounds__(1024) k_list_pairs(Views V, int cur, int off, int n, int which, int cap, int *pi,
                                                     int *pj, double *val, int *total)
{
    __shared__ int cnt[LIST_ONE_BLOCK];
    __shared__ int sums[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < n; k += 1024) {
        int id;
        const int c = count_row(V, cur, off, which, k, id);
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
    if (tid == 1023) *total = before + pre;
    for (int k = k0; k < k1; k++) {
        const int c = cnt[k];
        cnt[k] = at;
        at += c;
    }
    __syncthreads();
    if (cap > 0)
        for (int k = tid; k < n; k += 1024) write_row(V, cur, off, which, k, cnt, cap, pi, pj, val);
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

void launch_list_pairs(const Views &V, int cur, int off, int n, int which, int cap, int *pi, int *pj, double *val,
                       int *total, int *cnt, int *base, int *scan_scratch, cudaStream_t st)
{
    if (n <= LIST_ONE_BLOCK) {
        k_list_pairs<<<1, 1024, 0, st>>>(V, cur, off, n, which, cap, pi, pj, val, total);
        return;
    }
    const int grid = (n + 127) / 128 < 2048 ? (n + 127) / 128 : 2048;
    k_list_counts<<<grid, 128, 0, st>>>(V, cur, off, n, which, cnt);
    scan_excl(cnt, base, n, scan_scratch, st);
    cudaMemcpyAsync(total, base + n, sizeof(int), cudaMemcpyDeviceToDevice, st);
    if (cap > 0) k_list_fill<<<grid, 128, 0, st>>>(V, cur, off, n, which, base, cap, pi, pj, val);
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
