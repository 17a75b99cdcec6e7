// Bond creation on the device: the bonds of time step 1 (stepper.f90:93-101)
// with their geometry (bond_properties, bonds.f90:237-269), for the fields
// admitted to a batch fresh (not a restart) with cohesion on.
//
// Rule: every candidate pair i < j of a field (dist <= r_i + rtree, the
// reference's radius query) with deltan = (r_i + r_j) - dist >=
// -(bond_lim + bond_lim_rel (r_i + r_j)); with 0 < bond_frac < 1, only the
// pairs whose hash pair_hash32(bond_seed, i, j) / 2^32 is below bond_frac.
//
// At admission the fields' floes sit in their slots in reference order (slot
// = instance offset + reference id).  A cell list over the admitted floes
// gives each floe's neighbours without moving any state; one pass counts each
// floe's bonds, a scan places them, a second pass writes them in ascending
// partner id (the reference's j order in its bond loops) into the batch's
// bond table.  A group of eight lanes takes a floe: with one thread per floe
// the two passes took 64 us each on 4,096 floes, all of it one thread's chain
// of loads over some 25 cells.  Compiled with --fmad=false: distances and geometry round
// exactly as in the step and in the CPU oracle.
#include <algorithm>

#include "cells.cuh"
#include "kernels.h"

namespace godar {

// Floe s (slot = instance offset + reference id) against the floes of higher
// id of its field that fall to this lane: f(id of t, distance) for those the
// rule bonds to s.  The cell stencil (kx, ky) covers r_max + rtree + skin,
// beyond the candidate radius r_i + rtree.
template <class F>
GD_DEV void bi_partners(const Views &V, int side, const BondRule &R, const int *coff, const int *list, int s, int sub,
                        F f)
{
    const InstParams &P = V.P[V.inst[s]];
    const double xs = V.x[side][s], ys = V.y[side][s], rs = V.r[side][s];
    const int ids = s - P.off;
    const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
    const double Rc = rs + P.rtree;
    walk_cells(P, xs, ys, coff, sub, [&](int q) {
        const int t = list[q];
        const int idt = t - P.off;
        if (idt <= ids) return;
        const double dx = wrap_d(xs - V.x[side][t], P.nx, px);
        const double dy = wrap_d(ys - V.y[side][t], P.ny, py);
        const double dist = sqrt(dx * dx + dy * dy);
        if (!(dist <= Rc)) return;
        const double rt = V.r[side][t];
        const double deltan = (rs + rt) - dist;
        const double lim = R.lim + R.lim_rel * (rs + rt);
        bool sel = true;
        if (R.frac > 0.0 && R.frac < 1.0)
            sel = (double)pair_hash32((uint32_t)R.seed, (uint32_t)ids, (uint32_t)idt) * 0x1.0p-32 < R.frac;
        if (deltan >= -lim && sel) f(idt, dist);
    });
}

// Per admitted floe: the number of bonds it owns (it is the lower id), at
// cnt[s - s0]; zero for fields without fresh bonds.  Groups take the floes in
// the cell list's order.
__global__ void __launch_bounds__(256) k_bi_count(Views V, int side, int s0, int n, const BondRule *rule,
                                                  const int *coff, const int *list, int *cnt)
{
    const int sub = threadIdx.x & (GRP - 1), groups = gridDim.x * (blockDim.x / GRP);
    for (int k0 = blockIdx.x * (blockDim.x / GRP) + (threadIdx.x & ~31) / GRP; k0 < n; k0 += groups) {
        const int k = k0 + (threadIdx.x & 31) / GRP;
        int c = 0;
        if (k < n) {
            const BondRule R = rule[V.inst[list[k]]];
            if (R.fresh) bi_partners(V, side, R, coff, list, list[k], sub, [&](int, double) { c++; });
        }
#pragma unroll
        for (int o = GRP / 2; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (k < n && sub == 0) cnt[list[k] - s0] = c;
    }
}

// Bonds of each admitted field: the scanned counts at the field's first and
// last floe (first = the instance offset relative to s0).
__global__ void k_bi_totals(const int *scan, const int *first, const int *last, int m, int *tot)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m; k += gridDim.x * blockDim.x)
        tot[k] = scan[last[k]] - scan[first[k]];
}

// Bond q of the table, between floe s (the lower id) and reference id idt of
// its field, at distance dist.
GD_DEV void bi_write(const Views &V, int side, const InstParams &P, int s, int idt, double dist, int q, int *bond_hi,
                     BondStat *bstat, BondDyn *bdyn)
{
    const int t = P.off + idt;
    const double ri = V.r[side][s], hi = V.h[side][s], rj = V.r[side][t], hj = V.h[side][t];
    bond_hi[q] = idt;
    // bond_properties (bonds.f90:255-262)
    BondStat bs;
    bs.rb = P.lambda_rb * (ri < rj ? ri : rj);
    bs.hb = (hi + hj) / 2.0;
    bs.lb = dist;
    bs.sb = (2.0 * bs.rb) * bs.hb;
    bs.ib = ((2.0 / 3.0) * bs.hb) * ((bs.rb * bs.rb) * bs.rb);
    bs.pad = 0.0;
    // undamaged beam coefficients (bonds.f90:109-117) for the mixed path
    const double EA = P.eb * bs.sb, EI = P.eb * bs.ib, L = bs.lb;
    bs.k_ax = (float)(EA / L);
    bs.k_sh1 = (float)((12.0 * EI) / ((L * L) * L));
    bs.k_sh2 = (float)((6.0 * EI) / (L * L));
    bs.k_r1 = (float)((4.0 * EI) / L);
    bs.k_r2 = (float)((2.0 * EI) / L);
    bs.ei_l = (float)(EI / L);
    bs.ea_l = (float)(EA * L);
    bs.inv_l = (float)(1.0 / L);
    bstat[q] = bs;
    BondDyn d;
    d.dnb = 0.0; d.dtb = 0.0; d.thji = 0.0; d.thij = 0.0; d.dmg = 0.0;
    d.flag = 1;
    d.pad = 0;
    bdyn[q] = d;
}

// Writes floe s's bonds: bond_off of its global id, then its bonds in
// ascending partner id.  A group collects them in shared memory and places
// each by its rank; a floe with more than BI_CAP of them has its partners
// written with their distance (the distance slot lb of the static record),
// sorted in place and completed by one lane.
constexpr int BI_CAP = 64;
__global__ void __launch_bounds__(128) k_bi_fill(Views V, int side, int s0, int n, const BondRule *rule,
                                                 const int *coff, const int *list, const int *scan, int *bond_off,
                                                 int *bond_hi, BondStat *bstat, BondDyn *bdyn)
{
    __shared__ GroupBag<BI_CAP> bags[128 / GRP];
    const int sub = threadIdx.x & (GRP - 1), groups = gridDim.x * (blockDim.x / GRP);
    GroupBag<BI_CAP> &B = bags[threadIdx.x / GRP];
    for (int k0 = blockIdx.x * (blockDim.x / GRP) + (threadIdx.x & ~31) / GRP; k0 < n; k0 += groups) {
        const int k = k0 + (threadIdx.x & 31) / GRP;
        const int s = k < n ? list[k] : list[0];
        const int ig = V.inst[s];
        const BondRule R = rule[ig];
        const InstParams &P = V.P[ig];
        const bool on = k < n && R.fresh;
        // slot = global id for an admitted field; its bonds start at its
        // table offset plus the bonds of its lower ids
        const int b0 = on ? R.boff + (scan[s - s0] - scan[P.off - s0]) : 0;
        const int m = on ? scan[s - s0 + 1] - scan[s - s0] : 0;
        if (on && sub == 0) bond_off[s] = b0;
        if (sub == 0) B.n[0] = 0;
        __syncwarp();
        if (on && m <= BI_CAP) {
            bi_partners(V, side, R, coff, list, s, sub, [&](int idt, double dist) {
                const int q = atomicAdd(&B.n[0], 1);
                B.id[q] = idt;
                B.d[q] = dist;
            });
        } else if (on) {
            bi_partners(V, side, R, coff, list, s, sub, [&](int idt, double dist) {
                const int q = b0 + atomicAdd(&B.n[0], 1);
                bond_hi[q] = idt;
                bstat[q].lb = dist;
            });
        }
        __syncwarp();
        if (on && m <= BI_CAP) {
            for (int q = sub; q < m; q += GRP) {
                int at = 0;
                for (int j = 0; j < m; j++) at += B.id[j] < B.id[q];
                bi_write(V, side, P, s, B.id[q], B.d[q], b0 + at, bond_hi, bstat, bdyn);
            }
        } else if (on && sub == 0) {
            for (int a = 1; a < m; a++) {
                const int ja = bond_hi[b0 + a];
                const double da = bstat[b0 + a].lb;
                int b = a - 1;
                while (b >= 0 && bond_hi[b0 + b] > ja) {
                    bond_hi[b0 + b + 1] = bond_hi[b0 + b];
                    bstat[b0 + b + 1].lb = bstat[b0 + b].lb;
                    b--;
                }
                bond_hi[b0 + b + 1] = ja;
                bstat[b0 + b + 1].lb = da;
            }
            for (int a = 0; a < m; a++)
                bi_write(V, side, P, s, bond_hi[b0 + a], bstat[b0 + a].lb, b0 + a, bond_hi, bstat, bdyn);
        }
        __syncwarp();
    }
}

static int bi_grid(long long n, int block)
{
    return (int)std::max(1LL, std::min<long long>((n + block - 1) / block, 148LL * (2048 / block)));
}

void launch_bond_init_count(const Views &V, int side, int s0, int n, const BondRule *rule, const int *coff,
                            const int *list, int *scan_scratch, int *cnt, int *scan, cudaStream_t st)
{
    if (n <= 0) return;
    k_bi_count<<<bi_grid((long long)n * GRP, 256), 256, 0, st>>>(V, side, s0, n, rule, coff, list, cnt);
    scan_excl(cnt, scan, n, scan_scratch, st);
}

void launch_bond_init_totals(const int *scan, const int *first, const int *last, int m, int *tot, cudaStream_t st)
{
    if (m > 0) k_bi_totals<<<bi_grid(m, 128), 128, 0, st>>>(scan, first, last, m, tot);
}

void launch_bond_init_fill(const Views &V, int side, int s0, int n, const BondRule *rule, const int *coff,
                           const int *list, const int *scan, int *bond_off, int *bond_hi, BondStat *bstat,
                           BondDyn *bdyn, cudaStream_t st)
{
    if (n <= 0) return;
    k_bi_fill<<<bi_grid((long long)n * GRP, 128), 128, 0, st>>>(V, side, s0, n, rule, coff, list, scan, bond_off,
                                                                bond_hi, bstat, bdyn);
}

}  // namespace godar
