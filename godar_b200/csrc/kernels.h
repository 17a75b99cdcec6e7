// Host-side launch wrappers of the device kernels (build.cu, step_*.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"

namespace godar {

// Whether step kernels may be launched with programmatic dependent launch
// (GODAR_PDL=0: never).  Memory order is that of the stream either way,
// since every step kernel first waits for the kernel before it.
bool step_pdl();

// Launches a step kernel (one that starts with step_kernel_entry) on st,
// with programmatic dependent launch if pdl.
template <typename... Params, typename... Args>
inline void launch_step(bool pdl, void (*kern)(Params...), int grid, int block, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = 0;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&c, kern, args...);
}

// What destroyed engines left for later ones on the calling thread's context
// (streams, pinned memory, memory pools) back to the driver; whether there was
// any (engine.cu).
bool release_kept();

// The largest cluster an engine's kernels of whole steps may ask for: -1 before
// the first one (the attribute that allows more than eight blocks belongs to
// the kernel on one device, so every engine sets it), 0 where even eight were
// refused.
struct ClusterLimit { int blocks = -1; };

// The blocks of a kernel of whole steps (k_steps_fp64, k_steps_mixed): one, or
// a cluster of enough blocks to give every item a thread, at most SMALL_CLUSTER.
// One block finds what it wrote in its own L1 and its barrier takes 28 cycles;
// across blocks every phase starts from L2 behind a barrier of 380, and that
// costs less than another round of a block's threads over the pairs or the
// floes.  Us a step, one block against a cluster: 256 free floes FP64 5.0 and
// 7.5, mixed 4.2 and 6.5; 1,000 free mixed 11.0 and 6.5; 215 bonded FP64 (256
// pairs) 14.4 and 14.9, 230: 19.7 and 16.0; 256 bonded mixed 9.6 and 10.3, 270:
// 12.7 and 10.7.
inline int cluster_blocks(long long items, bool one)
{
    int blocks = 1;
    while (!one && blocks < SMALL_CLUSTER && (long long)blocks * SMALL_THREADS < items) blocks *= 2;
    return blocks;
}

// Launches it so.  A cluster that is refused is asked for with eight blocks,
// and then no more: false, with nothing launched.
template <typename... Params, typename... Args>
inline bool launch_cluster(ClusterLimit &most, bool pdl, void (*kern)(Params...), int want, cudaStream_t st,
                           Args... args)
{
    if (want > 1 && most.blocks < 0)
        most.blocks = cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                              cudaSuccess
                          ? SMALL_CLUSTER
                          : 8;
    while (want == 1 || most.blocks > 1) {
        const int blocks = want == 1 || want < most.blocks ? want : most.blocks;
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3((unsigned)blocks);
        c.blockDim = dim3(SMALL_THREADS);
        c.stream = st;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)blocks;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        c.attrs = at;
        c.numAttrs = pdl ? 2 : 1;
        if (cudaLaunchKernelEx(&c, kern, args...) == cudaSuccess) return true;
        cudaGetLastError();
        if (blocks == 1) return false;
        most.blocks = blocks > 8 ? 8 : 0;
    }
    return false;
}

void scan_excl(const int *in, int *out, int n, int *scratch, cudaStream_t st);
void radix_sort(uint32_t *keys, int *vals, uint32_t *keys_alt, int *vals_alt, int n, int bits,
                int *counts, int *scratch, cudaStream_t st);
// The cell list of floes [s0, s0 + n) over C cells: keys (n ints), the cells'
// offsets coff (C + 1), their floes (list, n, any order within a cell); cnt: C.
void launch_cell_list(const Views &V, int cur, int s0, int n, long long C, uint32_t *keys, int *cnt, int *coff,
                      int *list, int *scan_scratch, cudaStream_t st);
// The floes' state from side cur into cell order on the other side.
void launch_cell_place(const Views &V, int cur, const uint32_t *keys, const int *coff, const int *list,
                       const int *repack, int *old_slot, cudaStream_t st);
// The counts of every floe's partners (cnt: 2 N) and their scan (off2: 2 N + 1;
// off2[N] pairs), then the rows (lo_raw, up_raw: 8 and 16 bytes for every pair;
// row_max: raised to the partners of any floe with more than LONG_ROW).
constexpr int LONG_ROW = 192;
void launch_nbr_count(const Views &V, int side, const int *coff, int *cnt, int *off2, int *scan_scratch,
                      cudaStream_t st);
void launch_nbr_fill(const Views &V, int side, const int *coff, const int *off2, int up_by_id, int *lo_off,
                     int *up_off, int2 *ent_lo, int2 *ent_up, void *lo_raw, void *up_raw, int *row_max, cudaStream_t st);
void launch_rows_ready(int *status, int *nwork, unsigned *dsp, cudaStream_t st);
void launch_row_finish(const Views &V, int mixed, int side, const int *old_slot, const int *old_up_off,
                       const int2 *old_ent_up, const int *old_id, const void *old_hist, const int *up_off,
                       const int *lo_off, const int2 *ent_up, int2 *ent_lo, void *hist, int *bidx, unsigned *erow,
                       float *pdn, unsigned char *pfl, unsigned char *lfl, int *lo_of, const int *wfo,
                       cudaStream_t st);

// The FP64 time step: (b) every owner entry's distance and candidate test,
// with the pairs out of contact done there, and the pair physics of the work
// list, writing pair records and flags; the ordered sums of every floe's
// records and its ridging events, into FP64_FLOE_SUMS doubles per floe;
// (c)-(e) walls, forcing and the FP64 update (which also clears the work list).
constexpr int FP64_PAIR_REC_BYTES = 160;
constexpr int FP64_FLOE_SUMS = 18;
void launch_pairs_fp64(const Views &V, int cur, int n, const int *plist, const unsigned *erow, unsigned char *pfl,
                       FP64List L, void *rec, int block, cudaStream_t st);
void launch_pairs_list_fp64(const Views &V, int cur, int n, unsigned char *pfl, FP64List L, void *rec, int block,
                            cudaStream_t st);
// Diagnostic steps: the pairs of every owner entry (shelter: some field of the
// batch has sheltering).
void launch_pairs_diag_fp64(const Views &V, int cur, int E, int shelter, const unsigned *erow, unsigned char *pfl,
                            FP64List L, void *rec, cudaStream_t st);
// (light: no field of the batch has ridging, sheltering or walls)
void launch_row_sums_fp64(const Views &V, int cur, int diag, int light, const unsigned char *pfl, const void *rec,
                          const int *lo_n, const int *up_n, double *fs, int block, cudaStream_t st);
// At a rebuild: the pairs that can act on a step without diagnostics before
// the next one marked (listed[p]), every row reordered to hold them first
// (up_n / lo_n per floe), and the list of their owner-row positions for the
// screen (plist, pos[N] of them; pos: N + 1 ints; tmp: 2 E entries).
// Also sets the pairs' flags before the first step.
void launch_fp64_rows(const Views &V, int side, int E, const unsigned *erow, unsigned char *pfl,
                      unsigned char *listed, int *up_n, int *lo_n, int2 *tmp, int *pos, int *scan_scratch, int *plist, cudaStream_t st);
void launch_pairs_shel_fp64(const Views &V, int cur, int n, const int *plist, const unsigned *erow,
                            unsigned char *pfl, void *rec, cudaStream_t st);
void launch_group_sums_fp64(const Views &V, int cur, const unsigned char *pfl, const void *rec, const int *lo_n,
                            const int *up_n, double *fs, cudaStream_t st);
void launch_floes_fp64(const Views &V, int cur, int diag, int sic, int walls, int light, const double *fs, int *nwork, int block,
                       cudaStream_t st);
// At a rebuild: the bonds' working order (perm; wfo: N + 1, its first index of
// every slot) and working copies.  cnt: N.
void launch_fp64_bonds(const Views &V, int side, int *cnt, int *wfo, int *scan_scratch, int *perm, BondDyn *wdyn,
                       BondGeom64 *wgeo, cudaStream_t st);
// K whole steps of a small batch (n marked positions, E owner entries;
// shelter: some field of the batch has sheltering; drag: 8 N doubles; out:
// pinned host memory for the status word and the first expired step; done: an
// int that is zero): as one launch of one cluster up to ONE_CLUSTER_* items
// (positions, bonds and floes; one block where one_block_* says so), else, or
// where the cluster is refused and on large diagnostic steps (diag_apart), as
// two to four launches a step (one where no pair can act).  Returns the kernels
// launched.
constexpr int ONE_CLUSTER_FP64 = 1024, ONE_CLUSTER_MIXED = 4096;
// (FP64: no thread has a second floe or a second bond, nor a third item; mixed,
// where a pair is lighter: four rounds of items, in which a bond counts twice once
// there are two of floes; see cluster_blocks.  Floes in touch without bonds, one
// block and a cluster: 221 FP64 8.7 and 10.6 us a step, 271 mixed 10.6 and 13.8)
inline bool one_block_fp64(int N, int n, int NB)
{
    return N <= SMALL_THREADS && NB <= SMALL_THREADS && n + N <= 5 * SMALL_THREADS / 2;
}
inline bool one_block_mixed(int N, long long items, int NB)
{
    return N <= SMALL_THREADS ? items <= 4 * SMALL_THREADS : N <= 2 * SMALL_THREADS && items + NB <= 4 * SMALL_THREADS;
}
int launch_steps_fp64(const Views &V, ClusterLimit &most, int cur, int K, int diag_last, int base, int n, int E, int NB,
                       int shelter, int walls,
                       const int *plist, const unsigned *erow, unsigned char *pfl, void *rec, const int *lo_n,
                       const int *up_n, double *drag, FP64List L, int *out, int *done, cudaStream_t st);
// Whether a diagnostic step, which visits all E owner entries, leaves the launch
// of its chunk: a cluster has few threads, and the two launches of a step as
// many as there are entries.  A call of one such step: 400 floes with 5,214
// entries FP64 105 and 89 us, 2,299: 72 and 69; 2,000 floes with 700,000
// entries mixed 369 and 98, 1,000 with 13,000: 48 and 45.  FP64 sums walk their
// rows entry by entry, on one block through its L1: 85 floes, all candidates of
// one another, 107 and 128.
inline bool diag_apart(int N, int E, int blocks, bool fp64)
{
    return E > 4LL * blocks * SMALL_THREADS && !(fp64 && N <= SMALL_THREADS / 2);
}

// Whether a diagnostic step of the merged kernels sums its floes in a kernel of
// their own: the rows of every candidate are long, and the sums wait for them
// with the update's registers otherwise.  FP64 (which then leaves the pair
// physics to a work list too), a call, us, merged and apart: 60,000 bonded floes
// with six entries each 138 and 111, 41,250 without bonds 81 and 90; 30,000 with
// 351,000 entries 119 and 108, with 987,000 256 and 209; 20,000 with 240,000 96
// and 104; 5,000 with 1.2 M 1,073 and 1,108.
inline bool diag_sums_apart_fp64(int N, int E, int NB)
{
    return E + 4LL * NB > 10LL * N && (N > 32 * 1024 || (N > 8 * 1024 && E > 320 * 1024));
}
// Mixed, where the sums are short beside one long row (row_max: the most
// partners of a floe, 0 if no more than LONG_ROW): sums and update of 70,000
// floes of many sizes 139 and 85 us; a call of 51,476 alike sheltering ones 508
// and 627, of 112,870 with hardly a candidate each 62 and 69.
inline bool diag_sums_apart_mixed(int N, int E, int row_max)
{
    return N > 32 * 1024 && (long long)row_max * N > 16LL * E;
}

// How a plain step of the merged kernels sums the pairs of a floe: one thread
// a floe; by groups of lanes in the update's kernel, up to one wave of its
// blocks; by groups of lanes in a kernel of their own (sheltering fields, whose
// every candidate has a record).  rows: entries and bonds the sums walk; where
// there is hardly one a floe, seven of a group's lanes only wait (6,000 free
// floes FP64 9.5 us a step by groups and 8.3 by threads, mixed 8.1 and 7.8;
// bonded 18.8 and 21.6, 12.9 and 13.5).
enum GroupSums { SUMS_THREAD, SUMS_GROUP, SUMS_GROUP_APART };
inline GroupSums group_sums(int N, int shelter, long long rows)
{
    if (N <= 148 * 2 * GRP_FLOES) return shelter || 4 * rows > N ? SUMS_GROUP : SUMS_THREAD;
    return shelter ? SUMS_GROUP_APART : SUMS_THREAD;
}

// Mixed precision: pair and bond records (b, b'), summed per floe (c)-(e).
struct MixedBufs {
    unsigned char *pfl, *lfl;   // flags of the owner entries and of their mirror partner entries
    int *lo_of;                 // partner-row index of every owner entry
    float4 *rec;                // [2P] pair records: force/moments, shelter factors
    float2 *rx;                 // [P] ridging excesses of both floes
    float4 *pdg;                // [2P] diagnostic sums of the pair (diagnostic steps)
    float4 *brec, *bdg;         // [2NB], [4NB] bond records (per floe, slot order), diagnostic sums
    int *bfo;                   // [N+1] first bond record of every slot
    const BondGeom32 *bst;      // [NB] FP32 static bond records (working order)
    BondDyn *wdyn;              // [NB] dynamic bond records (working order)
    const int *winv;            // [NB] working index of every bond of the table
    const unsigned char *bfl_rd;   // [NB] live-bond flags at the start of the step
    unsigned char *bfl_wr;         // [NB] ... at its end (the other side)
    int4 *bsp;                  // [NB] slots of the bond's two floes, positions of their records (working order)
    float4 *fsum;               // [2N] per floe: fcx fcy mc fbx | fby mb shelter(air) shelter(water)
    float *frex;                // [N] per floe: ridging excess
    float4 *fdg;                // [2N] per floe, diagnostic steps: tac pc tab pb | sxx syy sxy syx
    unsigned *dsp;              // [4] displacement bound of the contact-list screening: per side,
                                // the largest squared step of any floe (FP32 bits, rounded up),
                                // then per side the cumulative bound D (FP32 bits); zero at a rebuild
};
void launch_pack_snap(const Views &V, int side, cudaStream_t st);
// The bonds' slots, record positions (bfo: N + 1) and working copies (perm:
// nb) of fresh rows.  cnt: N, blo: N + 1, list: nb, n2: 2 N, o2: 2 N + 1.
void launch_bond_lists(const Views &V, int side, int nb, int *slot_of, int4 *bsp, int *cnt, int *blo, int *list,
                       int *n2, int *o2, int *scan_scratch, int *bfo, int *perm, const BondStat *in,
                       const BondDyn *dyn, BondGeom32 *wst, BondDyn *wdyn, int4 *wsp, int *winv, unsigned char *wflag,
                       cudaStream_t st);
void launch_bond_work_scatter(const int *perm, int nb, const BondDyn *wdyn, BondDyn *dyn, cudaStream_t st);
void launch_pairs_screen(const Views &V, int cur, int diag, int P, int2 *eb, const int2 *stl,
                         MixedBufs B, int block, int variant, cudaStream_t st);
void launch_contact_list(const Views &V, int side, int P, const unsigned *erow, const unsigned char *pfl, int *mark,
                         int *pos, int *scan_scratch, int2 *eb, int2 *stl, const int *row_max, int *hs,
                         cudaStream_t st);
// Diagnostic steps: the pair physics of every owner entry.
void launch_pairs_diag(const Views &V, int cur, int P, const unsigned *erow_up, MixedBufs B, int block,
                       cudaStream_t st);
// light: no field of the batch has ridging, sheltering or walls; bounded: the
// pair kernel advances the displacement bound in every step since the rebuild.
void launch_floe_sums(const Views &V, int diag, int light, MixedBufs B, int block, cudaStream_t st);
void launch_pairs_shel_mixed(const Views &V, int cur, int n, int2 *eb, const int2 *stl, MixedBufs B, cudaStream_t st);
void launch_group_sums_mixed(const Views &V, MixedBufs B, cudaStream_t st);
void launch_bonds_mixed(const Views &V, int cur, int diag, int NB, MixedBufs B, int block, int variant,
                        unsigned test_spins, cudaStream_t st);
void launch_floes_mixed(const Views &V, int cur, int diag, int sic, int walls, int light, int bounded, MixedBufs B,
                        int block, cudaStream_t st);

// The same on the mixed path (n contact-list items eb/stl, bfl: the live-bond
// flags of both sides).
int launch_steps_mixed(const Views &V, ClusterLimit &most, int cur, int K, int diag_last, int base, int n, int E, int NB, int row_max,
                        int shelter, int walls, int ridging, int2 *eb, const int2 *stl, const unsigned *erow, unsigned char *bfl, MixedBufs B, int *out,
                        int *done, cudaStream_t st);

// Checkpoints: pair histories out and back in.
void launch_hist_list(const Views &V, int cur, int off, int n, int fp64, int hs, int *count, int *pi, int *pj,
                      double *h4, int cap, cudaStream_t st);
void launch_hist_inject(const Views &V, int cur, int off, int nh, const int *pi, const int *pj, const double *h4,
                        int *slot_of, int fp64, int hs, unsigned char *pfl, cudaStream_t st);

// Output helpers.  Field codes GODAR_F_*; GATHER_DTB1 .. + 3: the wall
// histories deltat_bc1, deltat_bc2, theta_bc1, theta_bc2.
constexpr int GATHER_DTB1 = 100;
void launch_set_forcing(InstParams *P, int ni, const double *uvw, cudaStream_t st);
void launch_gather_field(const Views &V, int cur, int inst, int off, int n, int field, double *out, cudaStream_t st);
// Several fields of the instance at slots [off, off + n) in id order, field q
// at out + q n.
struct FieldList { int n; int code[24]; };
void launch_gather_fields(const Views &V, int cur, int off, int n, const FieldList &F, double *out, cudaStream_t st);
// Per instance: momentum x, y, kinetic energy, largest speed (4 doubles).
void launch_instance_summary(const Views &V, int cur, double *out, cudaStream_t st);
// A pair list (0 candidates, 1 contacts, 2 live bonds) of the instance at
// slots [off, off + n), ascending in (i, j): its first cap pairs.  Returns where
// its length is written (total, or the end of base).  entries: of all the
// batch's rows that the list is made from; cnt, base: n + 1 ints each.
const int *launch_list_pairs(const Views &V, int cur, int off, int n, long long entries, int which, int cap, int *pi,
                             int *pj, double *val, int *total, int *cnt, int *base, int *scan_scratch,
                             cudaStream_t st);

// Batch relayout (membership changes), per field: its first new slot and bond,
// its first old ones (-1: admitted now).
struct RelayoutTable {
    int ni;
    const int *off, *old_off, *boff, *old_boff;
};
void launch_relayout_floes(const Views &Vo, int so, const Views &Vn, int sn, const RelayoutTable &T, int *inst,
                           int *repack, int n, cudaStream_t st);
void launch_relayout_bonds(const int *old_bond_off, int *new_bond_off, const int *inst, const int *old_hi,
                           const BondStat *old_st, const BondDyn *old_dy, int *new_hi, BondStat *new_st,
                           BondDyn *new_dy, const RelayoutTable &T, int n, int nb, cudaStream_t st);
void launch_set_int(int *p, int v, cudaStream_t st);
// hs[0..1] = status[0..1] (hs: pinned host memory), *base = next.
void launch_chunk_end(const int *status, int *hs, int *base, int next, cudaStream_t st);

// Bond creation at admission (bonds_init.cu): per-floe bond counts of the
// admitted floes [s0, s0 + n) on side `side` and their scan (coff, list: their
// cell list); per-field totals; the bond table's entries of the fresh fields.
void launch_bond_init_count(const Views &V, int side, int s0, int n, const BondRule *rule, const int *coff,
                            const int *list, int *scan_scratch, int *cnt, int *scan, cudaStream_t st);
void launch_bond_init_totals(const int *scan, const int *first, const int *last, int m, int *tot, cudaStream_t st);
void launch_bond_init_fill(const Views &V, int side, int s0, int n, const BondRule *rule, const int *coff,
                           const int *list, const int *scan, int *bond_off, int *bond_hi, BondStat *bstat,
                           BondDyn *bdyn, cudaStream_t st);

}  // namespace godar
