// One time step of every floe of a batch in FP64: the body of `stepper`
// (stepper.f90:44-343) as four kernels, bit-identical to the reference's
// sequential order.
//
//   k_pairs_fp64 (diagnostic steps: k_pairs_diag_fp64; sheltering fields:
//   k_step_pairs_shel_fp64, k_step_pairs_fp64), one thread per owner entry (pair of
//   candidates i < j by
//   id, stored in the row of the lower-id floe i): the FP64 distance of the
//   pair and the candidate test (dist <= r_i + rtree, stepper.f90:89-92);
//   pairs that need no pair physics and bonded pairs out of contact are done
//   there, the others go on a work list.
//
//   k_pairs_list_fp64, one thread per work-list entry: contact
//   (contact_forces.f90:1-87), ridging (ridging.f90:1-99), bond forces and
//   damage (bonds.f90:74-212), sheltering (forcing.f90:162-186) and the
//   stress magnitude (stepper.f90:238-271), computed ONCE per pair.  The
//   pair history and bond state are updated in place (one thread owns a
//   pair); what the two floes add to their sums goes to a record of the pair
//   (the operands of every sum term, not partial sums), written only when the
//   pair contributes anything.
//
//   k_row_sums_fp64, one thread per floe: sorts the floe's own row by
//   (distance, id) - the kd-tree's order, nearly sorted from the previous
//   step - then adds its pairs' records in the reference's order (partners
//   of lower id, ascending id, the floe as "j"; then its own row, the floe
//   as "i") with the same expressions as a sequential walk, so every FP64 sum
//   rounds as in the reference, and applies the pairs' ridging events in
//   that order (d).
//
//   k_floes_fp64, one thread per floe: its wall contacts (verify_bc,
//   boundaries.f90:1-97), drag, Coriolis and the shelter minimum (c,
//   forcing.f90:32-206), totals (stepper.f90:312-332) and the symplectic
//   Euler update (e, integration.f90:1-38).
//
// The kernels read the start-of-step floe state (side cur) and write side
// cur ^ 1.  No floe sum uses atomics, and no pair is evaluated twice.
#pragma once
#include "physics.cuh"

namespace godar {

// Bond w of the working order (by the slot of the lower-id floe, as the pairs
// are: a row's bonds are one stretch of memory).
GD_DEV void bond_load(const Views &V, int w, BondLocal &B)
{
    const BondDyn d = V.wdyn[w];
    const BondGeom64 c = V.wgeo[w];
    B.flag = d.flag;
    B.dmg = d.dmg; B.dnb = d.dnb; B.dtb = d.dtb; B.thji = d.thji; B.thij = d.thij;
    B.rb = c.rb; B.hb = c.hb; B.lb = c.lb; B.sb = c.sb; B.ib = c.ib;
}

GD_DEV void bond_store(const Views &V, int w, const BondLocal &B)
{
    BondDyn d;
    d.dnb = B.dnb; d.dtb = B.dtb; d.thji = B.thji; d.thij = B.thij; d.dmg = B.dmg;
    d.flag = B.flag;
    d.pad = 0;
    V.wdyn[w] = d;
}

// What one candidate pair adds to the sums of its two floes, in 32-byte
// groups: each group is written and read only when its flag says so (a
// bond on a plain step: the first and the third).
struct __align__(32) PairRec64 {
    double cosa, sina, ri_l, rj_l;     // any sum (PR_CONTACT, PR_BOND, PR_DIAG)
    double fcn, fcr, fct, mcc;         // PR_CONTACT
    double fbn, fbt, mji, mij;         // PR_BOND
    double ac, vol, sbt, S;            // diagnostic step: ac (contact), sbt (bond), S (PR_DIAG); vol: a ridging event
    double a_ij, a_ji, w_ij, w_ji;     // PR_SHEL
};

// Pair flags (one byte per pair, every owner entry writes its own).
enum : unsigned char {
    PR_CAND = 1,       // a candidate (dist <= r_i + rtree)
    PR_CONTACT = 2,
    PR_BOND = 4,       // a live bond after this step's breaking test
    PR_SHEL = 8,       // a shelter factor other than exactly 1
    PR_DIAG = 16,      // a stress term other than +-0 (diagnostic steps)
    PR_WHO1 = 32,      // ridging of the lower-id floe
    PR_WHO2 = 64,      // ridging of the higher-id floe
    PR_HIST = 128,     // the pair's tangential or rolling history may be nonzero (kept while not a candidate)
};

GD_DEV double stress_term(double S, double c1, double rl, double c2) { return ((S * c1) * rl) * c2; }

// reset_contact (reset.f90:1-15) of a candidate out of contact whose flags of
// the last step say that its tangential or rolling history may be nonzero.
// The flag spares every other pair the history's sector, read and written.
GD_DEV void reset_history(Hist4<double> *Hs, int p, unsigned old)
{
    if (old & PR_HIST) *(double2 *)&Hs[p] = make_double2(0.0, 0.0);
}

// A candidate without contact, bond or sheltering (old: its flags of the last
// step): its tangential and rolling histories are reset and, on a diagnostic
// step, its stress record and overlap written: pair_compute's normal, stress
// magnitude (no bond forces) and overlap, by the same expressions.  Returns
// the pair's flags.
template <bool DIAG>
GD_DEV unsigned quiet_candidate(const Views &V, Hist4<double> *Hs, int p, double dx, double dy, double dist,
                                double deltan, double ri, double rj, unsigned old, PairRec64 *rec)
{
    reset_history(Hs, p, old);
    unsigned f = PR_CAND;
    if (DIAG) {
        const double2 fc = *(const double2 *)&Hs[p].fcn;
        const double S = sqrt(fc.x * fc.x + fc.y * fc.y) + sqrt(0.0 * 0.0 + 0.0 * 0.0);
        const double cosa = -dx / dist, sina = -dy / dist;
        if (!(stress_term(S, cosa, ri, cosa) == 0.0 && stress_term(S, sina, ri, sina) == 0.0
              && stress_term(S, sina, ri, cosa) == 0.0 && stress_term(S, cosa, ri, sina) == 0.0)) {
            f |= PR_DIAG;
            PairRec64 &Q = rec[p];
            Q.cosa = cosa; Q.sina = sina; Q.ri_l = ri; Q.rj_l = rj;
            Q.S = S;
        }
        V.pdn[p] = (float)deltan;
    }
    return f;
}

// A sheltering field's candidate out of contact and without a bond, on a plain
// step (pair p, lower-id slot g, shapes' radii rg, rt): its histories are reset
// and its shelter factors computed, by pair_compute's expressions.  Returns the
// pair's flags.
GD_DEV unsigned sheltered_candidate(const Views &V, const InstParams &P, int cur, Hist4<double> *Hs, int p, int g,
                                    int t, double x, double y, double dx, double dy, double dist, double deltan,
                                    double rg, double rt, unsigned old, PairRec64 *rec)
{
    const Shape si = make_shape(P, rg, V.h[cur][g]), sj = make_shape(P, rt, V.h[cur][t]);
    double ua, va, uw, vw;
    wind_at(P, V.field, x, y, ua, va, uw, vw);
    const double cosa = -dx / dist, sina = -dy / dist;
    double a_ij, a_ji, w_ij, w_ji;
    shelter_pair<double>(si.hfa, sj.hfa, deltan, cosa, sina, ua, va, a_ij, a_ji);
    shelter_pair<double>(si.hfw, sj.hfw, deltan, cosa, sina, uw, vw, w_ij, w_ji);
    reset_history(Hs, p, old);
    if (a_ij == 1.0 && a_ji == 1.0 && w_ij == 1.0 && w_ji == 1.0) return PR_CAND;
    PairRec64 &Q = rec[p];
    Q.a_ij = a_ij; Q.a_ji = a_ji; Q.w_ij = w_ij; Q.w_ji = w_ji;
    return PR_CAND | PR_SHEL;
}

// Counts of a diagnostic step, per thread.
struct Counts64 { unsigned long long cand, cont, bond, plast; };

// The counts added to the counters (every lane of the warp calls it).
GD_DEV void add_counts(const Counts64 &C, unsigned long long *counters)
{
    unsigned long long c[4] = {C.cand, C.cont, C.bond, C.plast};
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c[q] += __shfl_down_sync(0xffffffffu, c[q], o);
        if ((threadIdx.x & 31) == 0 && c[q]) atomicAdd(&counters[q], c[q]);
    }
}

// The pair physics of one candidate (pair p, owner slot g, partner slot t,
// working bond bi or -1, offset dx, dy, flags `old` of the last step): history
// and bond in place, the record groups its flags name.  BONDS: for a bonded
// pair out of contact in a field without sheltering, the contact branch
// compiled out.  DIAG: a diagnostic step (stress records, overlaps, counts).
template <bool BONDS, bool DIAG>
GD_DEV void pair_work64(const Views &V, int cur, Hist4<double> *Hs, int p, int g, int t, int bi, double dx, double dy,
                        unsigned old, unsigned char *pfl, PairRec64 *rec, Counts64 &C)
{
    const InstParams &P = V.P[V.inst[g]];
    const bool shel = !BONDS && P.shelter != 0;
    const double r = V.r[cur][g];
    // the screen's distance, by the same expression
    const double dist = sqrt(dx * dx + dy * dy);
    BondLocal BL;
    if (bi >= 0) bond_load(V, bi, BL);
    // the history: a contact's, and on a diagnostic step the last contact
    // forces of every pair
    Hist4<double> H;
    H.deltat = H.thetarelc = H.fcn = H.fct = 0.0;
    if (DIAG || (!BONDS && (r + V.r[cur][t]) - dist > 0.0)) H = Hs[p];
    const Shape si = make_shape(P, r, V.h[cur][g]);
    const Shape sj = make_shape(P, V.r[cur][t], V.h[cur][t]);
    double ua = 0.0, va = 0.0, uw = 0.0, vw = 0.0;
    if (shel) wind_at(P, V.field, V.x[cur][g], V.y[cur][g], ua, va, uw, vw);
    const PairRes<double> R = pair_compute<double, !BONDS>(P, dx, dy, dist, V.u[cur][g], V.v[cur][g], V.om[cur][g],
                                                   V.u[cur][t], V.v[cur][t], V.om[cur][t], si, sj,
                                                   ua, va, uw, vw, H, bi >= 0 ? &BL : nullptr, shel);
    unsigned f = PR_CAND;
    if (R.contact) {
        Hs[p] = H;
        f |= PR_CONTACT;
        if (__double_as_longlong(H.deltat) | __double_as_longlong(H.thetarelc)) f |= PR_HIST;
    } else {
        reset_history(Hs, p, old);
    }
    if (bi >= 0) bond_store(V, bi, BL);

    if (R.bond_on) f |= PR_BOND;
    if (R.who == 1) f |= PR_WHO1;
    else if (R.who == 2) f |= PR_WHO2;
    if (shel && !(R.a_ij == 1.0 && R.a_ji == 1.0 && R.w_ij == 1.0 && R.w_ji == 1.0)) f |= PR_SHEL;
    // a stress term of +-0 leaves a sum unchanged (the sums start at +0
    // and never become -0), so only nonzero ones (NaN included) count
    if (DIAG && !(stress_term(R.S, R.cosa, R.ri_l, R.cosa) == 0.0 && stress_term(R.S, R.sina, R.ri_l, R.sina) == 0.0
                  && stress_term(R.S, R.sina, R.ri_l, R.cosa) == 0.0
                  && stress_term(R.S, R.cosa, R.ri_l, R.sina) == 0.0))
        f |= PR_DIAG;
    PairRec64 &Q = rec[p];
    if (f & (PR_CONTACT | PR_BOND | PR_DIAG)) {
        Q.cosa = R.cosa; Q.sina = R.sina; Q.ri_l = R.ri_l; Q.rj_l = R.rj_l;
    }
    if (f & PR_CONTACT) {
        Q.fcn = R.fcn; Q.fcr = R.fcr; Q.fct = R.fct; Q.mcc = R.mcc;
        if (DIAG) Q.ac = R.ac;
    }
    if (f & (PR_WHO1 | PR_WHO2)) Q.vol = R.vol;
    if (f & PR_BOND) {
        Q.fbn = R.fbn; Q.fbt = R.fbt; Q.mji = R.mji; Q.mij = R.mij;
        if (DIAG) Q.sbt = R.sbt;
    }
    if (f & PR_DIAG) Q.S = R.S;
    if (f & PR_SHEL) { Q.a_ij = R.a_ij; Q.a_ji = R.a_ji; Q.w_ij = R.w_ij; Q.w_ji = R.w_ji; }
    pfl[p] = (unsigned char)f;
    if (DIAG) {
        V.pdn[p] = (float)R.deltan;
        C.cand++;
        C.cont += R.contact;
        C.bond += R.bond_on;
        C.plast += R.who != 0;
    }
}

// Owner entries on a plain step of a batch without sheltering: the FP64
// distance (kept for the row sort), the candidate test, and every pair that is
// not in contact.
// A non-candidate keeps its history and bond state.  A candidate without a
// bond is a quiet_candidate.  A bonded one goes through the pair physics with
// the contact branch compiled out.  The others go on the work list with
// their slots, bond index and offset.
// It visits the positions of plist only (n of them: the pairs that can act
// before the next rebuild, see k_fp64_mark; nine in ten are bonded on the
// benchmark's fields); a diagnostic step visits every owner entry
// (k_pairs_diag_fp64, k_step_pairs_fp64<true>).
// Latency bounds it (half its warps' registers are the bond's FP64 chain), so
// what it waits for is kept short: the screen and the bonds were two kernels
// with a 32-byte item a bond between them, each gathering both floes, the bond
// state in reference order, and every pair's history read and written back.
// 529,113 floes, 0.82 M bonds: 41 + 84 us then, 77 us now.
__global__ void __launch_bounds__(128, 6) k_pairs_fp64(Views V, int cur, int n, const int *plist, const unsigned *erow,
                                                    unsigned char *pfl, FP64List L, PairRec64 *rec)
{
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    Hist4<double> *Hs = (Hist4<double> *)V.hist[0];   // in place: one thread per pair
    Counts64 C = {0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const int stride = gridDim.x * blockDim.x;
    // every lane of a warp runs the same iterations (the list append is warp-wide)
    for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
        const int i = i0 + lane;
        const bool on = i < n;
        // lanes past the end read item 0 and store nothing
        const int e = plist[on ? i : 0];
        const int g = (int)erow[e];
        const int2 en = V.ent_up[e];
        const int t = en.x, p = en.y;
        const InstParams &P = V.P[V.inst[g]];
        const double rg = V.r[cur][g], rt = V.r[cur][t];
        const int bi = V.bidx[p];
        const unsigned old = pfl[p];
        const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
        const double dx = wrap_d(V.x[cur][g] - V.x[cur][t], P.nx, px);
        const double dy = wrap_d(V.y[cur][g] - V.y[cur][t], P.ny, py);
        const double dist = sqrt(dx * dx + dy * dy);
        const double deltan = (rg + rt) - dist;
        const bool cand = on && dist <= rg + P.rtree;
        const bool heavy = cand && deltan > 0.0;
        if (on) V.edist[e] = dist;
        const unsigned m = __ballot_sync(0xffffffffu, heavy);
        if (m) {
            int base = 0;
            if (lane == 0) base = atomicAdd(L.n, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (heavy) {
                FP64Item it;
                it.p = p; it.g = g; it.t = t; it.bi = bi;
                it.dx = dx; it.dy = dy;
                L.work[base + __popc(m & ((1u << lane) - 1))] = it;
            }
        }
        if (!on || heavy) continue;
        if (!cand) {
            // history and bond state stay as they are
            pfl[p] = (unsigned char)(old & PR_HIST);
        } else if (bi >= 0) {
            pair_work64<true, false>(V, cur, Hs, p, g, t, bi, dx, dy, old, pfl, rec, C);
        } else {
            pfl[p] = (unsigned char)quiet_candidate<false>(V, Hs, p, dx, dy, dist, deltan, rg, rt, old, rec);
        }
    }
}

// The pairs of a diagnostic step of a batch without sheltering: every owner
// entry (n of them), most of which are candidates out of contact, with the pair
// physics of the others left to the work list.  Few registers, so that many
// entries' loads wait side by side: a call of one such step, this and the list
// against one kernel of both: 130,000 floes of many sizes 299 and 372 us,
// 300,000 526 and 666, 600,000 bonded 577 and 659.
__global__ void __launch_bounds__(128, 12) k_pairs_diag_fp64(Views V, int cur, int n, const unsigned *erow,
                                                             unsigned char *pfl, FP64List L, PairRec64 *rec)
{
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    Hist4<double> *Hs = (Hist4<double> *)V.hist[0];   // in place: one thread per pair
    Counts64 C = {0, 0, 0, 0};
    const int lane = threadIdx.x & 31;
    const int stride = gridDim.x * blockDim.x;
    // every lane of a warp runs the same iterations (the list append is warp-wide)
    for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
        const int e = i0 + lane;
        bool heavy = false;
        FP64Item it;
        if (e < n) {
            const int g = (int)erow[e];
            const int2 en = V.ent_up[e];
            const int t = en.x, p = en.y;
            const InstParams &P = V.P[V.inst[g]];
            const double rg = V.r[cur][g], rt = V.r[cur][t];
            const int bi = V.bidx[p];
            const unsigned old = pfl[p];
            const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
            const double dx = wrap_d(V.x[cur][g] - V.x[cur][t], P.nx, px);
            const double dy = wrap_d(V.y[cur][g] - V.y[cur][t], P.ny, py);
            const double dist = sqrt(dx * dx + dy * dy);
            const double deltan = (rg + rt) - dist;
            V.edist[e] = dist;
            if (!(dist <= rg + P.rtree)) {
                // history and bond state stay as they are
                pfl[p] = (unsigned char)(old & PR_HIST);
                V.pdn[p] = __int_as_float(0x7fc00000);
            } else if (deltan > 0.0 || bi >= 0) {
                heavy = true;
                it.p = p; it.g = g; it.t = t; it.bi = bi;
                it.dx = dx; it.dy = dy;
            } else {
                pfl[p] = (unsigned char)quiet_candidate<true>(V, Hs, p, dx, dy, dist, deltan, rg, rt, old, rec);
                C.cand++;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, heavy);
        if (m) {
            int base = 0;
            if (lane == 0) base = atomicAdd(L.n, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (heavy) L.work[base + __popc(m & ((1u << lane) - 1))] = it;
        }
    }
    __syncwarp();
    add_counts(C, V.counters);
}

// The work list: contacts (on a diagnostic step bonds too).
template <bool DIAG>
__global__ void __launch_bounds__(128, 4) k_pairs_list_fp64(Views V, int cur, FP64List L, unsigned char *pfl,
                                                         PairRec64 *rec)
{
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    Hist4<double> *Hs = (Hist4<double> *)V.hist[0];   // in place: one thread per pair
    Counts64 C = {0, 0, 0, 0};
    const int stride = gridDim.x * blockDim.x;
    const int n = *(volatile const int *)L.n;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        // the pair, both slots, the bond index and the pair's offset come along
        const FP64Item w = L.work[k];
        pair_work64<false, DIAG>(V, cur, Hs, w.p, w.g, w.t, w.bi, w.dx, w.dy, pfl[w.p], pfl, rec, C);
    }
    __syncwarp();
    if (DIAG) add_counts(C, V.counters);
}

// The pair result one floe's sums need, from the pair's record.  A group the
// flags leave out holds values that make its terms no-ops: no contact, no
// bond, shelter factors of exactly 1 (what the pair computed), stress of 0.
GD_DEV double4 load_group(const double *q)
{
    const double2 u = ((const double2 *)q)[0], v = ((const double2 *)q)[1];
    return make_double4(u.x, u.y, v.x, v.y);
}

GD_DEV PairRes<double> rec_load(const PairRec64 *rec, int p, unsigned f, bool diag)
{
    PairRes<double> R;
    R.contact = (f & PR_CONTACT) != 0;
    R.bond_on = (f & PR_BOND) != 0;
    R.cosa = R.sina = R.ri_l = R.rj_l = 0.0;
    R.fcn = R.fcr = R.fct = R.mcc = R.ac = 0.0;
    R.fbn = R.fbt = R.mji = R.mij = R.sbt = 0.0;
    R.a_ij = R.a_ji = R.w_ij = R.w_ji = 1.0;
    R.S = 0.0;
    R.vol = 0.0;
    R.who = (f & PR_WHO1) ? 1 : (f & PR_WHO2) ? 2 : 0;
    const PairRec64 &Q = rec[p];
    if (f & (PR_CONTACT | PR_BOND | PR_DIAG)) {
        const double4 q = load_group(&Q.cosa);
        R.cosa = q.x; R.sina = q.y; R.ri_l = q.z; R.rj_l = q.w;
    }
    if (f & PR_CONTACT) {
        const double4 q = load_group(&Q.fcn);
        R.fcn = q.x; R.fcr = q.y; R.fct = q.z; R.mcc = q.w;
        if (diag) R.ac = Q.ac;
    }
    if (R.who) R.vol = Q.vol;
    if (f & PR_BOND) {
        const double4 q = load_group(&Q.fbn);
        R.fbn = q.x; R.fbt = q.y; R.mji = q.z; R.mij = q.w;
        if (diag) R.sbt = Q.sbt;
    }
    if (f & PR_DIAG) R.S = Q.S;
    if (f & PR_SHEL) {
        const double4 q = load_group(&Q.a_ij);
        R.a_ij = q.x; R.a_ji = q.y; R.w_ij = q.z; R.w_ji = q.w;
    }
    return R;
}

// Per-floe outputs of the row sums, [FS64_COUNT][N] doubles (the last eight
// on diagnostic steps only).
enum {
    FS64_FCX, FS64_FCY, FS64_MC, FS64_FBX, FS64_FBY, FS64_MB, FS64_HSFA, FS64_HSFW, FS64_R, FS64_H,
    FS64_TAC, FS64_PC, FS64_TAB, FS64_PB, FS64_SXX, FS64_SYY, FS64_SXY, FS64_SYX, FS64_COUNT
};

// Adds one pair's record to the sums of a floe: `LO` - a partner of lower id
// (the floe is "j"), else one of its own partners ("i").
template <bool DIAG, bool LO>
GD_DEV void add_pair(const PairRec64 *rec, int p, unsigned f, const InstParams &P, Acc<double> &A, Shape &run,
                     bool shel)
{
    if (!f) return;
    const PairRes<double> R = rec_load(rec, p, f, DIAG);
    if (LO) {
        acc_side_j(A, R, P.lambda_lb, shel, DIAG);
        if (R.who == 2) apply_dh(P, run, R.vol);
    } else {
        acc_side_i(A, R, P.lambda_lb, shel, DIAG);
        if (R.who == 1) apply_dh(P, run, R.vol);
    }
}

// Adds the pair records of row entries [e0, e1) of a floe in order.  Flags
// and entries are fetched four at a time so that their loads overlap; the
// sums themselves run strictly in row order.
template <bool DIAG, bool LO>
GD_DEV void row_sum(const int2 *ent, int e0, int e1, const unsigned char *pfl, const PairRec64 *rec,
                    const InstParams &P, Acc<double> &A, Shape &run, bool shel)
{
    for (int e = e0; e < e1; e += 4) {
        int pk[4];
        unsigned fk[4];
#pragma unroll
        for (int k = 0; k < 4; k++) pk[k] = e + k < e1 ? ent[e + k].y : -1;
#pragma unroll
        for (int k = 0; k < 4; k++) fk[k] = pk[k] >= 0 ? pfl[pk[k]] & ~PR_HIST : 0u;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (fk[k]) add_pair<DIAG, LO>(rec, pk[k], fk[k], P, A, run, shel);
    }
}

// Sorts owner-row entries [a0, a1) into the kd-tree's order: ascending
// distance, ties by id.  Rows are nearly sorted from the previous step, so
// insertion sort is linear.
GD_DEV void sort_own(const Views &V, int cur, int a0, int a1)
{
    for (int a = a0 + 1; a < a1; a++) {
        const double da = V.edist[a];
        double db = V.edist[a - 1];
        if (db < da) continue;
        const int2 ea = V.ent_up[a];
        const int ida = V.id[cur][ea.x];
        int b = a - 1;
        while (b >= a0) {
            db = V.edist[b];
            if (db < da || (db == da && V.id[cur][V.ent_up[b].x] < ida)) break;
            V.ent_up[b + 1] = V.ent_up[b];
            V.edist[b + 1] = db;
            b--;
        }
        V.ent_up[b + 1] = ea;
        V.edist[b + 1] = da;
    }
}

// The ordered sums of floe g's pairs' records (A) and its shape after its
// pairs' ridging events, in the reference's order (partners of lower id in
// ascending id, then its own row in the kd-tree's order).  Every row holds
// first the pairs that can act on a step without diagnostics before the next
// rebuild (lo_n / up_n of them), then the others, each part in the row's
// order: a plain step walks the first part only; a diagnostic step, on which
// every candidate adds its stress, walks both parts merged.
template <bool DIAG>
GD_DEV Shape row_sums64(const Views &V, int cur, int g, const InstParams &P, const unsigned char *pfl,
                        const PairRec64 *rec, const int *lo_n, const int *up_n, Acc<double> &A)
{
    const bool shel = P.shelter != 0;
    A.fcx = A.fcy = A.mc = A.fbx = A.fby = A.mb = 0.0;
    A.tac = A.pc = A.tab = A.pb = 0.0;
    A.sxx = A.syy = A.sxy = A.syx = 0.0;
    A.hsfa = A.hsfw = shel ? 1.0 : 0.0;
    Shape run = make_shape(P, V.r[cur][g], V.h[cur][g]);
    const int l0 = V.lo_off[g], l1 = V.lo_off[g + 1], lm = l0 + lo_n[g];
    const int el = V.up_off[g], e1 = V.up_off[g + 1], em = el + up_n[g];

    if (!DIAG) {
        row_sum<false, true>(V.ent_lo, l0, lm, pfl, rec, P, A, run, shel);
        sort_own(V, cur, el, em);
        row_sum<false, false>(V.ent_up, el, em, pfl, rec, P, A, run, shel);
    } else {
        // ---- partners of lower id (the floe is the reference's "j"):
        // the two parts merged by ascending id
        int a = l0, b = lm;
        int ida = a < lm ? V.id[cur][V.ent_lo[a].x] : 0, idb = b < l1 ? V.id[cur][V.ent_lo[b].x] : 0;
        while (a < lm || b < l1) {
            int take;
            if (b >= l1 || (a < lm && ida < idb)) {
                take = a++;
                if (a < lm) ida = V.id[cur][V.ent_lo[a].x];
            } else {
                take = b++;
                if (b < l1) idb = V.id[cur][V.ent_lo[b].x];
            }
            const int p = V.ent_lo[take].y;
            add_pair<true, true>(rec, p, pfl[p] & ~PR_HIST, P, A, run, shel);
        }
        // ---- own row (the floe is "i"): each part sorted, merged by
        // (distance, id)
        sort_own(V, cur, el, em);
        sort_own(V, cur, em, e1);
        a = el;
        b = em;
        while (a < em || b < e1) {
            bool first = b >= e1;
            if (!first && a < em) {
                const double da = V.edist[a], db = V.edist[b];
                first = da < db || (da == db && V.id[cur][V.ent_up[a].x] < V.id[cur][V.ent_up[b].x]);
            }
            const int p = V.ent_up[first ? a++ : b++].y;
            add_pair<true, false>(rec, p, pfl[p] & ~PR_HIST, P, A, run, shel);
        }
    }
    return run;
}

// Floes [0, N), first part: the ordered sums.
template <bool DIAG, bool LIGHT>
__global__ void __launch_bounds__(128) k_row_sums_fp64(Views V, int cur, const unsigned char *pfl,
                                                       const PairRec64 *rec, const int *lo_n, const int *up_n,
                                                       double *fs)
{
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    const size_t N = (size_t)V.N;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < V.N; g += gridDim.x * blockDim.x) {
        const InstParams &P = V.P[V.inst[g]];
        Acc<double> A;
        const Shape run = row_sums64<DIAG>(V, cur, g, P, pfl, rec, lo_n, up_n, A);
        fs[FS64_FCX * N + g] = A.fcx; fs[FS64_FCY * N + g] = A.fcy; fs[FS64_MC * N + g] = A.mc;
        fs[FS64_FBX * N + g] = A.fbx; fs[FS64_FBY * N + g] = A.fby; fs[FS64_MB * N + g] = A.mb;
        if (!LIGHT) {
            fs[FS64_HSFA * N + g] = A.hsfa; fs[FS64_HSFW * N + g] = A.hsfw;
            fs[FS64_R * N + g] = run.r; fs[FS64_H * N + g] = run.h;
        }
        if (DIAG) {
            fs[FS64_TAC * N + g] = A.tac; fs[FS64_PC * N + g] = A.pc;
            fs[FS64_TAB * N + g] = A.tab; fs[FS64_PB * N + g] = A.pb;
            fs[FS64_SXX * N + g] = A.sxx; fs[FS64_SYY * N + g] = A.syy;
            fs[FS64_SXY * N + g] = A.sxy; fs[FS64_SYX * N + g] = A.syx;
        }
    }
}

// The sums of one floe on a plain step by a group of GRP lanes.  One thread
// per floe spends its time on a chain of loads a row entry long (row, flag,
// record), and a step waits for its longest row: a large floe among small
// ones, or any row of a sheltering field, whose every candidate has a record
// (measured on 512 floes of such a field: 36 us of a 48 us step).  Here the
// lanes load entries, flags and records side by side.
//
// The order of every sum is row_sums64's.  Only pairs in contact or bonded
// add to the force sums: they are listed in shared memory, the partner row's
// in row order, the own row's ranked by (distance, id), and their records are
// then added one after the other, each handed round from the lane that loaded
// it; every lane of the group holds the same sums.  A shelter factor only
// lowers a minimum, whose result does not depend on the order as long as no
// factor is NaN; each lane keeps its own and they are merged at the end.  A
// floe with a NaN factor, or with more than CAP pairs to list, goes the
// sequential way on the group's first lane.
constexpr int GRP_CAP = 24;

struct GroupList {
    double d[GRP_CAP];
    int p[GRP_CAP], id[GRP_CAP];
    int q[GRP_CAP];               // pair index by rank
    unsigned char f[GRP_CAP], fq[GRP_CAP];
};

GD_DEV double shfl_grp(double v, int src) { return __shfl_sync(0xffffffffu, v, src, GRP); }

// on: whether this group has a floe (g); every lane of the warp calls.  The
// result is valid in the group's first lane.
GD_DEV void group_sums64(const Views &V, int cur, bool on, int g, const unsigned char *pfl, const PairRec64 *rec,
                         const int *lo_n, const int *up_n, GroupList &L, Acc<double> &A, Shape &run)
{
    const int lane = threadIdx.x & 31, sub = lane & (GRP - 1);
    const unsigned gmask = ((1u << GRP) - 1u) << (lane & ~(GRP - 1)), below = (1u << lane) - 1u;
    const InstParams &P = V.P[on ? V.inst[g] : 0];
    const bool shel = P.shelter != 0;
    A.fcx = A.fcy = A.mc = A.fbx = A.fby = A.mb = 0.0;
    A.hsfa = A.hsfw = shel ? 1.0 : 0.0;
    int e0[2] = {0, 0}, e1[2] = {0, 0};
    if (on) {
        run = make_shape(P, V.r[cur][g], V.h[cur][g]);
        e0[0] = V.lo_off[g]; e1[0] = e0[0] + lo_n[g];
        e0[1] = V.up_off[g]; e1[1] = e0[1] + up_n[g];
    }
    int m = 0, mlo = 0;             // pairs listed, of the partner row
    bool seq = false;
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const int2 *ent = side ? V.ent_up : V.ent_lo;
        for (int b = e0[side]; __any_sync(0xffffffffu, b < e1[side]); b += GRP) {
            const int e = b + sub;
            int p = 0, id = 0;
            unsigned f = 0;
            double d = 0.0;
            if (e < e1[side]) {
                const int2 en = ent[e];
                p = en.y;
                f = pfl[p];
                if (side) {
                    d = V.edist[e];
                    id = V.id[cur][en.x];
                }
            }
            if (f & PR_SHEL) {
                const double4 q = load_group(&rec[p].a_ij);
                const double fa = side ? q.y : q.x, fw = side ? q.w : q.z;
                seq |= fa != fa || fw != fw;
                A.hsfa = tmin(A.hsfa, fa);
                A.hsfw = tmin(A.hsfw, fw);
            }
            const bool add = (f & (PR_CONTACT | PR_BOND)) != 0;
            const unsigned bal = __ballot_sync(0xffffffffu, add) & gmask;
            const int k = m + __popc(bal & below);
            if (add && k < GRP_CAP) {
                L.p[k] = p; L.f[k] = (unsigned char)f;
                L.d[k] = d; L.id[k] = id;
            }
            m += __popc(bal);
        }
        if (side == 0) mlo = m;
    }
    seq = (__ballot_sync(0xffffffffu, seq) & gmask) != 0 || m > GRP_CAP;
    if (seq) m = mlo = 0;
    __syncwarp();
    // the own row's pairs by (distance, id)
    for (int k = sub; k < m; k += GRP) {
        int at = k;
        if (k >= mlo) {
            at = mlo;
            for (int j = mlo; j < m; j++) at += L.d[j] < L.d[k] || (L.d[j] == L.d[k] && L.id[j] < L.id[k]);
        }
        L.q[at] = L.p[k];
        L.fq[at] = L.f[k];
    }
    __syncwarp();
    for (int b = 0; __any_sync(0xffffffffu, b < m); b += GRP) {
        double4 qa, qb;
        qa = qb = make_double4(0.0, 0.0, 0.0, 0.0);
        if (b + sub < m) {
            const PairRec64 &Q = rec[L.q[b + sub]];
            qa = load_group(&Q.cosa);
            qb = load_group(L.fq[b + sub] & PR_CONTACT ? &Q.fcn : &Q.fbn);
        }
        for (int j = 0; j < GRP && __any_sync(0xffffffffu, b + j < m); j++) {
            PairRes<double> R;
            R.cosa = shfl_grp(qa.x, j); R.sina = shfl_grp(qa.y, j);
            R.ri_l = shfl_grp(qa.z, j); R.rj_l = shfl_grp(qa.w, j);
            const double bx = shfl_grp(qb.x, j), by = shfl_grp(qb.y, j);
            const double bz = shfl_grp(qb.z, j), bw = shfl_grp(qb.w, j);
            if (b + j >= m) continue;
            const unsigned f = L.fq[b + j];
            const int p = L.q[b + j];
            R.contact = (f & PR_CONTACT) != 0;
            R.bond_on = (f & PR_BOND) != 0;
            if (R.contact) { R.fcn = bx; R.fcr = by; R.fct = bz; R.mcc = bw; }
            if (R.bond_on) {
                R.fbn = bx; R.fbt = by; R.mji = bz; R.mij = bw;
                if (R.contact) {
                    const double4 q = load_group(&rec[p].fbn);
                    R.fbn = q.x; R.fbt = q.y; R.mji = q.z; R.mij = q.w;
                }
            }
            if (b + j < mlo) {
                acc_side_j(A, R, P.lambda_lb, false, false);
                if (f & PR_WHO2) apply_dh(P, run, rec[p].vol);
            } else {
                acc_side_i(A, R, P.lambda_lb, false, false);
                if (f & PR_WHO1) apply_dh(P, run, rec[p].vol);
            }
        }
    }
#pragma unroll
    for (int o = GRP / 2; o > 0; o >>= 1) {
        A.hsfa = tmin(A.hsfa, __shfl_xor_sync(0xffffffffu, A.hsfa, o));
        A.hsfw = tmin(A.hsfw, __shfl_xor_sync(0xffffffffu, A.hsfw, o));
    }
    if (seq && on && sub == 0) run = row_sums64<false>(V, cur, g, P, pfl, rec, lo_n, up_n, A);
    __syncwarp();
}

// Floe g, second part: walls with the shape after the floe's pair events
// (run), drag and Coriolis with the final shape, totals and the FP64 update
// of step sic of a chunk (base: the chunk's first global step number, -1: in
// device memory).  The shape after the events is make_shape of its radius and
// thickness (apply_dh ends with make_shape too).  drag: the floe's drag and
// Coriolis terms computed ahead with its start-of-step shape (eight planes;
// null: none), taken if no event changed the shape.  LIGHT: a batch without
// ridging, sheltering and walls: the shape stays, equal on both sides, and is
// not written.  Returns the wall events.
template <bool DIAG, bool WALLS, bool LIGHT = false>
GD_DEV int floe_update64(const Views &V, int cur, int base, int sic, int g, const InstParams &P, const Acc<double> &A,
                         Shape run, const double *drag)
{
    const int nxt = cur ^ 1;
    const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
    const double x = V.x[cur][g], y = V.y[cur][g], th = V.th[cur][g];
    const double u = V.u[cur][g], v = V.v[cur][g], om = V.om[cur][g];
    const double r0 = V.r[cur][g], h0 = V.h[cur][g];

    // ---- walls with the shape after this floe's pair events (a batch
    // without walls neither reads nor writes the wall histories, which are
    // zero on both sides)
    WallOut W;
    int wev = 0;
    if (WALLS) {
        double dtb1 = V.dtb1[cur][g], dtb2 = V.dtb2[cur][g];
        double thb1 = V.thb1[cur][g], thb2 = V.thb2[cur][g];
        verify_bc(P, x, y, u, v, om, run, dtb1, dtb2, thb1, thb2, W, wev);
        V.dtb1[nxt][g] = dtb1; V.dtb2[nxt][g] = dtb2;
        V.thb1[nxt][g] = thb1; V.thb2[nxt][g] = thb2;
    } else {
        W.fx_bc = W.fy_bc = W.m_bc = 0.0;
        W.sxx = W.syy = W.sxy = W.syx = 0.0;
        W.ta_bc = W.p_bc = 0.0;
    }

    // ---- drag and Coriolis with the final shape
    Drag<double> D;
    if (drag && run.r == r0 && run.h == h0) {
        const size_t N = (size_t)V.N;
        D.fax = drag[0 * N + g]; D.fay = drag[1 * N + g]; D.fwx = drag[2 * N + g]; D.fwy = drag[3 * N + g];
        D.ma = drag[4 * N + g]; D.mw = drag[5 * N + g]; D.fcorx = drag[6 * N + g]; D.fcory = drag[7 * N + g];
    } else {
        double ua, va, uw, vw;
        wind_at(P, V.field, x, y, ua, va, uw, vw);
        D = forcing<double>(P, run, u, v, om, ua, va, uw, vw, A.hsfa, A.hsfw);
    }

    // ---- totals and integration (FP64)
    const double fcx = A.fcx, fcy = A.fcy, fbx = A.fbx, fby = A.fby, mc = A.mc, mb = A.mb;
    const double fax = D.fax, fay = D.fay, fwx = D.fwx, fwy = D.fwy;
    const double tfx = ((((fcx + fbx) + fax) + fwx) + D.fcorx) + W.fx_bc;
    const double tfy = ((((fcy + fby) + fay) + fwy) + D.fcory) + W.fy_bc;
    const double mt = (((mc + mb) + D.ma) + D.mw) + W.m_bc;
    const double dt = P.dt;
    const double u1 = u + (tfx / run.mass) * dt;
    const double v1 = v + (tfy / run.mass) * dt;
    const double om1 = om + (mt / run.inertia) * dt;
    double x1 = x + u1 * dt;
    double y1 = y + v1 * dt;
    const double th1 = th + om1 * dt;
    if (px) { if (x1 < 0.0) x1 = x1 + P.nx; else if (x1 >= P.nx) x1 = x1 - P.nx; }
    if (py) { if (y1 < 0.0) y1 = y1 + P.ny; else if (y1 >= P.ny) y1 = y1 - P.ny; }
    V.x[nxt][g] = x1; V.y[nxt][g] = y1; V.th[nxt][g] = th1;
    V.u[nxt][g] = u1; V.v[nxt][g] = v1; V.om[nxt][g] = om1;
    if (!LIGHT) { V.r[nxt][g] = run.r; V.h[nxt][g] = run.h; }

    // ---- neighbour-list validity and finiteness
    const double ddx = wrap_d(x1 - V.x0[cur][g], P.nx, px), ddy = wrap_d(y1 - V.y0[cur][g], P.ny, py);
    const double half = 0.5 * P.skin;
    if (ddx * ddx + ddy * ddy > half * half) {
        atomicOr(V.status, ST_EXPIRED);
        atomicMin(V.expired_at, base >= 0 ? base + sic : global_step(V, sic));
    }
    if (!(isfinite(x1) && isfinite(y1) && isfinite(u1) && isfinite(v1) && isfinite(om1) && isfinite(th1)))
        atomicOr(V.status, ST_NAN);

    if (DIAG) {
        const size_t N = (size_t)V.N;
        const double rr = run.r;
        const double sxx = (A.sxx + W.sxx) + (fax + fwx) * rr;
        const double syy = (A.syy + W.syy) + (fay + fwy) * rr;
        const double sxy = (A.sxy + W.sxy) + 0.0;
        const double syx = (A.syx + W.syx) + 0.0;
        const double tac = A.tac, tab = A.tab;
        const double pa = tac != 0.0 ? A.pc / tac : 0.0;
        const double pbv = tab != 0.0 ? A.pb / tab : 0.0;
        const double pw = W.ta_bc != 0.0 ? W.p_bc / W.ta_bc : 0.0;
        double *D0 = V.diag;
        D0[0 * N + g] = tfx; D0[1 * N + g] = tfy; D0[2 * N + g] = fcx; D0[3 * N + g] = fcy;
        D0[4 * N + g] = fbx; D0[5 * N + g] = fby; D0[6 * N + g] = mt; D0[7 * N + g] = mc;
        D0[8 * N + g] = mb; D0[9 * N + g] = sxx; D0[10 * N + g] = syy; D0[11 * N + g] = sxy;
        D0[12 * N + g] = syx; D0[13 * N + g] = (pa + pbv) + pw;
    }
    return DIAG ? wev : 0;
}

// Floes [0, N), second part, from the sums of the first.
// Memory bounds both parts.  The LIGHT instances (a batch without ridging,
// sheltering and walls) leave out what then stays as it was: the shape and the
// sheltering factors.  529,113 floes: sums 69 -> 60 us, update 44 -> 39 (the
// same by each field's own options: 69 and 49, its loads wait for the options).
template <bool DIAG, bool WALLS, bool LIGHT>
__global__ void __launch_bounds__(128) k_floes_fp64(Views V, int cur, int sic, const double *fs, int *nwork)
{
    step_kernel_entry();
    // the work list was used by the pair kernels before this one
    if (blockIdx.x == 0 && threadIdx.x == 0) *nwork = 0;
    if (floe_update_stopped(V, -1, sic)) return;
    const size_t N = (size_t)V.N;
    unsigned long long n_plast = 0;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < V.N; g += gridDim.x * blockDim.x) {
        const InstParams &P = V.P[V.inst[g]];
        Acc<double> A;
        A.fcx = fs[FS64_FCX * N + g]; A.fcy = fs[FS64_FCY * N + g]; A.mc = fs[FS64_MC * N + g];
        A.fbx = fs[FS64_FBX * N + g]; A.fby = fs[FS64_FBY * N + g]; A.mb = fs[FS64_MB * N + g];
        A.hsfa = LIGHT ? 0.0 : fs[FS64_HSFA * N + g];
        A.hsfw = LIGHT ? 0.0 : fs[FS64_HSFW * N + g];
        if (DIAG) {
            A.tac = fs[FS64_TAC * N + g]; A.pc = fs[FS64_PC * N + g];
            A.tab = fs[FS64_TAB * N + g]; A.pb = fs[FS64_PB * N + g];
            A.sxx = fs[FS64_SXX * N + g]; A.syy = fs[FS64_SYY * N + g];
            A.sxy = fs[FS64_SXY * N + g]; A.syx = fs[FS64_SYX * N + g];
        }
        const Shape run = LIGHT ? make_shape(P, V.r[cur][g], V.h[cur][g])
                                : make_shape(P, fs[FS64_R * N + g], fs[FS64_H * N + g]);
        n_plast += floe_update64<DIAG, WALLS, LIGHT>(V, cur, -1, sic, g, P, A, run, nullptr);
    }

    if (DIAG) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) n_plast += __shfl_down_sync(0xffffffffu, n_plast, o);
        if ((threadIdx.x & 31) == 0 && n_plast) atomicAdd(&V.counters[3], n_plast);
    }
}

// ---------------------------------------------------------------- small batches
// A batch of few floes is bound by the latency of one thread's dependent
// loads and FP64 operations and by the gaps between kernels, not by any
// rate.  k_steps_fp64 runs a chunk of K whole steps in one launch of one
// cluster (or one block): the screen and the pair physics of every entry in
// one pass, each thread carrying its pair from the distance to the record,
// beside the drag and Coriolis terms of every floe (they need the pairs only
// where an event changes the shape or in a sheltering field, where the update
// computes them again); a cluster barrier; the ordered sums and the update of
// every floe; a cluster barrier.  Two barriers a step stand in for four
// kernels.  Every value is computed by the functions the four kernels use.
struct SmallArgs64 {
    int cur, K, diag_last, base;   // first side, steps, diagnostics on the last one, global number of the first
    int n, E;                      // marked positions (plist), owner entries
    const int *plist;
    const unsigned *erow;
    unsigned char *pfl;
    PairRec64 *rec;
    const int *lo_n, *up_n;
    double *drag;                  // [8][N]
    int nd;                        // floes whose drag the pair kernel computes: N or 0
    int *out;                      // pinned host memory: the status word and the first expired step
    int *done;                     // blocks of k_step_floes_fp64 that have finished
};

// One owner entry: k_pairs_fp64 and k_pairs_list_fp64 in one.
template <bool DIAG>
GD_DEV void pair_entry64(const Views &V, int cur, int e, const unsigned *erow, unsigned char *pfl, PairRec64 *rec,
                         Counts64 &C)
{
    Hist4<double> *Hs = (Hist4<double> *)V.hist[0];
    const int g = (int)erow[e];
    const int2 en = V.ent_up[e];
    const int t = en.x, p = en.y;
    const InstParams &P = V.P[V.inst[g]];
    const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
    const double rg = V.r[cur][g], rt = V.r[cur][t];
    const int bi = V.bidx[p];
    const unsigned old = pfl[p];
    const double dx = wrap_d(V.x[cur][g] - V.x[cur][t], P.nx, px);
    const double dy = wrap_d(V.y[cur][g] - V.y[cur][t], P.ny, py);
    const double dist = sqrt(dx * dx + dy * dy);
    V.edist[e] = dist;
    if (!(dist <= rg + P.rtree)) {
        // history and bond state stay as they are
        pfl[p] = (unsigned char)(old & PR_HIST);
        if (DIAG) V.pdn[p] = __int_as_float(0x7fc00000);
        return;
    }
    const double deltan = (rg + rt) - dist;
    if (deltan > 0.0 || P.shelter != 0 || bi >= 0) {
        pair_work64<false, DIAG>(V, cur, Hs, p, g, t, bi, dx, dy, old, pfl, rec, C);
    } else {
        pfl[p] = (unsigned char)quiet_candidate<DIAG>(V, Hs, p, dx, dy, dist, deltan, rg, rt, old, rec);
        if (DIAG) C.cand++;
    }
}

// The drag and Coriolis terms of floe g with its start-of-step shape, unless
// its field has sheltering (which needs the pairs first).
GD_DEV void drag_ahead64(const Views &V, int cur, int g, double *drag)
{
    const InstParams &P = V.P[V.inst[g]];
    if (P.shelter != 0) return;
    const size_t N = (size_t)V.N;
    double ua, va, uw, vw;
    wind_at(P, V.field, V.x[cur][g], V.y[cur][g], ua, va, uw, vw);
    const Drag<double> D = forcing<double>(P, make_shape(P, V.r[cur][g], V.h[cur][g]), V.u[cur][g], V.v[cur][g],
                                           V.om[cur][g], ua, va, uw, vw, 0.0, 0.0);
    drag[0 * N + g] = D.fax; drag[1 * N + g] = D.fay; drag[2 * N + g] = D.fwx; drag[3 * N + g] = D.fwy;
    drag[4 * N + g] = D.ma; drag[5 * N + g] = D.mw; drag[6 * N + g] = D.fcorx; drag[7 * N + g] = D.fcory;
}

template <bool DIAG>
GD_DEV void small_pairs64(const Views &V, const SmallArgs64 &A, int cur)
{
    const int nthr = gridDim.x * blockDim.x;
    const int n = DIAG ? A.E : A.n;
    const int n0 = (n + 31) & ~31;      // the floes start on a warp of their own
    Counts64 C = {0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n0 + A.nd; i += nthr) {
        if (i < n) {
            pair_entry64<DIAG>(V, cur, DIAG ? i : A.plist[i], A.erow, A.pfl, A.rec, C);
        } else if (i >= n0) {
            drag_ahead64(V, cur, i - n0, A.drag);
        }
    }
    __syncwarp();
    if (DIAG) add_counts(C, V.counters);
}

// The floes' sums and update, one thread per floe.
template <bool DIAG, bool WALLS>
GD_DEV void small_floes64(const Views &V, const SmallArgs64 &A, int cur, int sic)
{
    const int nthr = gridDim.x * blockDim.x;
    Counts64 C = {0, 0, 0, 0};
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < V.N; g += nthr) {
        const InstParams &P = V.P[V.inst[g]];
        Acc<double> S;
        const Shape run = row_sums64<DIAG>(V, cur, g, P, A.pfl, A.rec, A.lo_n, A.up_n, S);
        C.plast += floe_update64<DIAG, WALLS>(V, cur, A.base, sic, g, P, S, run, P.shelter != 0 ? nullptr : A.drag);
    }
    __syncwarp();
    if (DIAG) add_counts(C, V.counters);
}

__global__ void __launch_bounds__(SMALL_THREADS, 1) k_steps_fp64(Views V, SmallArgs64 A)
{
    step_kernel_entry();
    for (int k = 0; k < A.K; k++) {
        // the same answer in every thread: the status is written between the
        // two barriers of a step only
        if (*(volatile int *)V.status & ST_ABORT) break;
        const int cur = A.cur ^ (k & 1);
        const bool diag = A.diag_last && k == A.K - 1;
        if (diag) small_pairs64<true>(V, A, cur);
        else small_pairs64<false>(V, A, cur);
        cluster_sync();
        if (diag) small_floes64<true, true>(V, A, cur, k);
        else small_floes64<false, true>(V, A, cur, k);
        cluster_sync();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) publish_status(V, A.out);
}

// The two halves of a step as ordinary grids, for batches with more work
// than one cluster does quickly: two launches a step instead of four.  The
// second one of a chunk's last step publishes the status word.
// MINB blocks an SM: a sheltering pair is a chain of dependent FP64
// instructions and loads (the FP64 pipe 15% busy at 182 registers and two
// blocks), so items that fill more than one wave of two blocks run four, at
// the price of a few spills: 65,536 sheltering floes 195 -> 145 us.
template <bool DIAG, int MINB>
__global__ void __launch_bounds__(128, MINB) k_step_pairs_fp64(Views V, SmallArgs64 A, int cur)
{
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    small_pairs64<DIAG>(V, A, cur);
}

// The pairs of a plain step of a sheltering batch whose items fill several
// rounds of one wave: out of contact and without a bond a pair needs its
// shelter factors only, and such pairs stay on their lane; the others (one in
// five of a packed field's, in nearly every warp) collect in shared memory and
// go through the physics 32 at a time, so that a warp does not run it for a few
// lanes.  65,536 floes: 198 -> 143 us a step; 9,473 (little more than one wave
// of items) as without.
constexpr int SHEL_THREADS = 128, SHEL_WAVE = 148 * 4 * SHEL_THREADS;
__global__ void __launch_bounds__(SHEL_THREADS, 4) k_step_pairs_shel_fp64(Views V, SmallArgs64 A, int cur)
{
    struct Item { int p, g, t, bi; double dx, dy; unsigned old; };
    __shared__ Item list[SHEL_THREADS / 32][64];
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    Hist4<double> *Hs = (Hist4<double> *)V.hist[0];
    Item *const L = list[threadIdx.x / 32];
    const int lane = threadIdx.x & 31, nthr = gridDim.x * blockDim.x;
    const unsigned lt = (1u << lane) - 1u;
    Counts64 C = {0, 0, 0, 0};
    int waiting = 0;
    // every lane of a warp runs the same iterations
    for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < A.n; i0 += nthr) {
        bool heavy = false;
        Item it;
        if (i0 + lane < A.n) {
            const int e = A.plist[i0 + lane];
            const int g = (int)A.erow[e];
            const int2 en = V.ent_up[e];
            const int t = en.x, p = en.y;
            const InstParams &P = V.P[V.inst[g]];
            const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
            const double rg = V.r[cur][g], rt = V.r[cur][t];
            const int bi = V.bidx[p];
            const unsigned old = A.pfl[p];
            const double x = V.x[cur][g], y = V.y[cur][g];
            const double dx = wrap_d(x - V.x[cur][t], P.nx, px), dy = wrap_d(y - V.y[cur][t], P.ny, py);
            const double dist = sqrt(dx * dx + dy * dy);
            V.edist[e] = dist;
            const double deltan = (rg + rt) - dist;
            if (!(dist <= rg + P.rtree)) {
                // history and bond state stay as they are
                A.pfl[p] = (unsigned char)(old & PR_HIST);
            } else if (deltan > 0.0 || bi >= 0) {
                heavy = true;
                it.p = p; it.g = g; it.t = t; it.bi = bi;
                it.dx = dx; it.dy = dy; it.old = old;
            } else if (P.shelter != 0) {
                A.pfl[p] = (unsigned char)sheltered_candidate(V, P, cur, Hs, p, g, t, x, y, dx, dy, dist, deltan, rg,
                                                              rt, old, A.rec);
            } else {
                A.pfl[p] = (unsigned char)quiet_candidate<false>(V, Hs, p, dx, dy, dist, deltan, rg, rt, old, A.rec);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, heavy);
        if (heavy) L[waiting + __popc(m & lt)] = it;
        waiting += __popc(m);
        __syncwarp();
        if (waiting >= 32 || i0 + nthr >= A.n) {
            const int k = max(waiting - 32, 0);
            if (k + lane < waiting) {
                it = L[k + lane];
                pair_work64<false, false>(V, cur, Hs, it.p, it.g, it.t, it.bi, it.dx, it.dy, it.old, A.pfl, A.rec, C);
            }
            waiting = k;
            __syncwarp();
        }
    }
    if (lane < waiting) {
        const Item it = L[lane];
        pair_work64<false, false>(V, cur, Hs, it.p, it.g, it.t, it.bi, it.dx, it.dy, it.old, A.pfl, A.rec, C);
    }
    // the drag of the floes out of sheltering fields (a small batch's update
    // takes it from here)
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < A.nd; g += nthr)
        drag_ahead64(V, cur, g, A.drag);
}

template <bool DIAG, bool WALLS>
__global__ void __launch_bounds__(128) k_step_floes_fp64(Views V, SmallArgs64 A, int cur, int sic)
{
    step_kernel_entry();
    if (!floe_update_stopped(V, A.base, sic)) small_floes64<DIAG, WALLS>(V, A, cur, sic);
    if (sic == A.K - 1) publish_status_last(V, A.done, A.out);
}

// The second half of a plain step with the floes' sums by groups of lanes: a
// block sums GRP_FLOES floes, then gives every floe's update a thread.
__global__ void __launch_bounds__(SMALL_THREADS, 2) k_step_floes_grp_fp64(Views V, SmallArgs64 A, int cur, int sic)
{
    __shared__ GroupList list[GRP_FLOES];
    __shared__ double sum[10][GRP_FLOES];
    __shared__ int stopped;
    step_kernel_entry();
    // one answer per block: another block may raise an expiry meanwhile
    if (threadIdx.x == 0) stopped = floe_update_stopped(V, A.base, sic);
    __syncthreads();
    const int grp = threadIdx.x / GRP;
    for (int g0 = blockIdx.x * GRP_FLOES; !stopped && g0 < V.N; g0 += gridDim.x * GRP_FLOES) {
        const bool on = g0 + grp < V.N;
        Acc<double> S;
        Shape run;
        run.r = run.h = 0.0;
        group_sums64(V, cur, on, g0 + grp, A.pfl, A.rec, A.lo_n, A.up_n, list[grp], S, run);
        if (on && threadIdx.x % GRP == 0) {
            sum[0][grp] = S.fcx; sum[1][grp] = S.fcy; sum[2][grp] = S.mc;
            sum[3][grp] = S.fbx; sum[4][grp] = S.fby; sum[5][grp] = S.mb;
            sum[6][grp] = S.hsfa; sum[7][grp] = S.hsfw;
            sum[8][grp] = run.r; sum[9][grp] = run.h;
        }
        __syncthreads();
        const int q = threadIdx.x, g = g0 + q;
        if (q < GRP_FLOES && g < V.N) {
            const InstParams &P = V.P[V.inst[g]];
            S.fcx = sum[0][q]; S.fcy = sum[1][q]; S.mc = sum[2][q];
            S.fbx = sum[3][q]; S.fby = sum[4][q]; S.mb = sum[5][q];
            S.hsfa = sum[6][q]; S.hsfw = sum[7][q];
            run = make_shape(P, sum[8][q], sum[9][q]);
            floe_update64<false, true>(V, cur, A.base, sic, g, P, S, run, P.shelter != 0 ? nullptr : A.drag);
        }
        __syncthreads();
    }
    if (sic == A.K - 1) publish_status_last(V, A.done, A.out);
}

// The sums of a plain step by groups of lanes as a kernel of their own, for
// sheltering batches of more floes than one wave of the kernel above: they
// wait for loads, and without the update's registers four blocks an SM wait
// side by side instead of two.  18,945 sheltering floes: 93 -> 66 us a step;
// 65,536: 253 -> 198, of which the pairs' denser blocks give 50.
__global__ void __launch_bounds__(SMALL_THREADS, 4) k_group_sums_fp64(Views V, int cur, const unsigned char *pfl,
                                                                      const PairRec64 *rec, const int *lo_n,
                                                                      const int *up_n, double *fs)
{
    __shared__ GroupList list[GRP_FLOES];
    step_kernel_entry();
    if (*(volatile int *)V.status & ST_ABORT) return;
    const size_t N = (size_t)V.N;
    const int grp = threadIdx.x / GRP;
    for (int g0 = blockIdx.x * GRP_FLOES; g0 < V.N; g0 += gridDim.x * GRP_FLOES) {
        const int g = g0 + grp;
        const bool on = g < V.N;
        Acc<double> S;
        Shape run;
        run.r = run.h = 0.0;
        group_sums64(V, cur, on, g, pfl, rec, lo_n, up_n, list[grp], S, run);
        if (on && threadIdx.x % GRP == 0) {
            fs[FS64_FCX * N + g] = S.fcx; fs[FS64_FCY * N + g] = S.fcy; fs[FS64_MC * N + g] = S.mc;
            fs[FS64_FBX * N + g] = S.fbx; fs[FS64_FBY * N + g] = S.fby; fs[FS64_MB * N + g] = S.mb;
            fs[FS64_HSFA * N + g] = S.hsfa; fs[FS64_HSFW * N + g] = S.hsfw;
            fs[FS64_R * N + g] = run.r; fs[FS64_H * N + g] = run.h;
        }
    }
}

// ... and the update from them, as the last kernel of a small batch's step; on
// a diagnostic step from k_row_sums_fp64's.
template <bool DIAG, bool WALLS>
__global__ void __launch_bounds__(64) k_step_update_fp64(Views V, SmallArgs64 A, int cur, int sic, const double *fs,
                                                         int *nwork)
{
    step_kernel_entry();
    // the work list was used by the pair kernels before this one
    if (DIAG && blockIdx.x == 0 && threadIdx.x == 0) *nwork = 0;
    const size_t N = (size_t)V.N;
    Counts64 C = {0, 0, 0, 0};
    if (!floe_update_stopped(V, A.base, sic))
        for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < V.N; g += gridDim.x * blockDim.x) {
            const InstParams &P = V.P[V.inst[g]];
            Acc<double> S;
            S.fcx = fs[FS64_FCX * N + g]; S.fcy = fs[FS64_FCY * N + g]; S.mc = fs[FS64_MC * N + g];
            S.fbx = fs[FS64_FBX * N + g]; S.fby = fs[FS64_FBY * N + g]; S.mb = fs[FS64_MB * N + g];
            S.hsfa = fs[FS64_HSFA * N + g]; S.hsfw = fs[FS64_HSFW * N + g];
            if (DIAG) {
                S.tac = fs[FS64_TAC * N + g]; S.pc = fs[FS64_PC * N + g];
                S.tab = fs[FS64_TAB * N + g]; S.pb = fs[FS64_PB * N + g];
                S.sxx = fs[FS64_SXX * N + g]; S.syy = fs[FS64_SYY * N + g];
                S.sxy = fs[FS64_SXY * N + g]; S.syx = fs[FS64_SYX * N + g];
            }
            const Shape run = make_shape(P, fs[FS64_R * N + g], fs[FS64_H * N + g]);
            C.plast += floe_update64<DIAG, WALLS>(V, cur, A.base, sic, g, P, S, run,
                                                  P.shelter != 0 ? nullptr : A.drag);
        }
    __syncwarp();
    if (DIAG) add_counts(C, V.counters);
    if (sic == A.K - 1) publish_status_last(V, A.done, A.out);
}

}  // namespace godar
