// Initial-condition generator on the GPU: places disks of given radii in a
// rectangular domain without overlap (random sequential addition with
// relaxation), for the dense polydisperse fields the benchmark
// configurations need.  The reference builds its initial fields with
// tools/init/gridded_placement.py:111-313 (a jittered lattice written as
// files/{x,y,r,h}<n>.dat, one value per line); the fields placed here are
// written in that format by generators.Field.write_reference_inputs.
//
// Disks are placed largest first, in radius classes (class c holds radii in
// [rmin 2^c, rmin 2^(c+1))).  For a class, the grid's cells are twice the
// class's largest radius, every disk already placed is entered into each
// cell its bounding box meets, and rounds repeat until the class is placed:
//   1. every unplaced disk of the class draws random positions (a
//      counter-based generator of seed, disk, round and attempt) and relaxes
//      each one by pushing it out of the placed disks it overlaps (the sum of
//      the overlaps, 12 iterations), keeping the first position that is free;
//   2. a free position is kept if no free position of a disk of the class
//      with a lower index overlaps it (the others retry next round).
// Every list is ordered (disks by index within a cell), so a placement
// depends only on its inputs and seed.
//
// What bounds a round is not any rate but the chain of one disk's attempts
// (8 positions of 12 iterations, each over up to four cells) and the host
// between the kernels.  A warp takes a disk, four lanes an attempt, so its
// eight positions relax side by side and four placed disks are tested at once;
// the cell lists are built by counting (their places by a scan, the order in
// a cell restored by a sort of its few entries), which needs no length on the
// host; all memory is drawn once; and the host reads one number a round.
// 32,768 disks at 66 %: 39-50 ms with one thread per disk, radix sorts and
// allocations per round, 9-11 ms so; 65,536 polydisperse ones 61 and 16 ms.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/godar_gpu.h"
#include "common.cuh"
#include "cover.h"
#include "kernels.h"

namespace godar {
namespace {

struct PGrid {
    int ncx, ncy;
    double cwx, cwy, Lx, Ly;
    int px, py;
};

GD_DEV uint64_t mix64(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

GD_DEV double uni(uint64_t &s)
{
    s += 0x9e3779b97f4a7c15ULL;
    return (double)(mix64(s) >> 11) * 0x1.0p-53;
}

GD_DEV double pwrap(double d, double L, int per)
{
    if (!per) return d;
    if (d > 0.5 * L) d -= L;
    else if (d < -0.5 * L) d += L;
    return d;
}

GD_DEV int wrapc(int c, int nc, int per) { return per ? ((c % nc) + nc) % nc : c; }

// A placed disk as a cell's list holds it.
struct __align__(32) Cover {
    double x, y, r;
    int j, pad;
};

// Coverage of the placed disks: one entry per cell that a placed disk's
// bounding box meets, counted (FILL = false) and written (true; cnt: how many
// of each cell's entries are still to come).  The first `big` disks, which may
// meet more than COVER_ALONE cells each, are spread over the whole grid.
constexpr double COVER_ALONE = 4096.0;
template <bool FILL>
__global__ void k_cover(int n, int big, const double *x, const double *y, const double *r,
                        const unsigned char *placed, PGrid G, int *cnt, const int *off, int *list)
{
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
    for (int i = 0; i < n; i++) {
        int first = tid, stride = nthr;
        if (i >= big) {
            // from here on a thread per disk
            i = max(i, big + tid);
            if (i >= n) break;
            first = 0;
            stride = 1;
        }
        if (placed[i]) {
            int ax, bx, ay, by;
            cell_span(x[i] - r[i], x[i] + r[i], G.cwx, G.ncx, G.px, ax, bx);
            cell_span(y[i] - r[i], y[i] + r[i], G.cwy, G.ncy, G.py, ay, by);
            const int w = max(0, bx - ax + 1), cells = w * max(0, by - ay + 1);
            for (int k = first; k < cells; k += stride) {
                const int c = wrapc(ay + k / w, G.ncy, G.py) * G.ncx + wrapc(ax + k % w, G.ncx, G.px);
                if (FILL) list[off[c] + atomicSub(&cnt[c], 1) - 1] = i;
                else atomicAdd(&cnt[c], 1);
            }
        }
        if (i >= big) i += nthr - 1;
    }
}

// Every cell's entries in ascending index, with their disks.
__global__ void k_cover_order(int ncell, const int *off, int *list, const double *x, const double *y, const double *r,
                              Cover *cov)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
        const int a = off[c], b = off[c + 1];
        for (int k = a + 1; k < b; k++) {
            const int v = list[k];
            int q = k;
            while (q > a && list[q - 1] > v) {
                list[q] = list[q - 1];
                q--;
            }
            list[q] = v;
        }
        for (int k = a; k < b; k++) {
            const int j = list[k];
            Cover e;
            e.x = x[j]; e.y = y[j]; e.r = r[j];
            e.j = j; e.pad = 0;
            cov[k] = e;
        }
    }
}

// Whether wrapped cell coordinate w lies in the span [a, b] of cell_span.
GD_DEV bool in_span(int w, int a, int b, int nc, int per)
{
    if (!per) return w >= a && w <= b;
    if (b - a + 1 >= nc) return true;
    return ((w - a) % nc + nc) % nc <= b - a;
}

// Step 1: free positions of the unplaced disks [c0, c1), a warp per disk, four
// lanes per attempt.  A candidate spans at most 2 x 2 cells (cells are at
// least twice the class's largest radius); a placed disk met in several of
// them is counted in the first.  The lanes of an attempt test a cell's
// entries four at a time; the pushes are added in the entries' order.  The
// disk takes the free position of its first successful attempt, so an attempt
// after a successful one stops.
constexpr int ATTEMPTS = 8;
__global__ void __launch_bounds__(256) k_trial(int c0, int c1, const double *r, const unsigned char *placed, PGrid G,
                                               const int *off, const Cover *cov, uint64_t seed, int round,
                                               unsigned char *cand, double *tx, double *ty)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 3, att = lane >> 2, quad = lane & ~3;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int i = c0 + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < c1; i += warps) {
        const double rad = r[i];
        const double xlo = G.px ? 0.0 : rad, xhi = G.px ? G.Lx : G.Lx - rad;
        const double ylo = G.py ? 0.0 : rad, yhi = G.py ? G.Ly : G.Ly - rad;
        if (placed[i] || !(xhi > xlo && yhi > ylo)) {
            if (lane == 0) cand[i] = 0;
            continue;
        }
        uint64_t s = mix64(seed ^ (0x632be59bd9b4e019ULL * (uint64_t)(i + 1))) ^ mix64((uint64_t)round + 1);
        // attempt a takes the generator's values 2 a and 2 a + 1
        s += 2 * (uint64_t)att * 0x9e3779b97f4a7c15ULL;
        double cx = xlo + (xhi - xlo) * uni(s);
        double cy = ylo + (yhi - ylo) * uni(s);
        bool live = true, found = false;
        for (int it = 0; it < 12; it++) {
            int ax = 0, bx = -1, ay = 0, by = -1;
            if (live) {
                cell_span(cx - rad, cx + rad, G.cwx, G.ncx, G.px, ax, bx);
                cell_span(cy - rad, cy + rad, G.cwy, G.ncy, G.py, ay, by);
            }
            const int nxs = min(bx - ax + 1, 2), nys = min(by - ay + 1, 2);
            const int wx0 = wrapc(ax, G.ncx, G.px), wx1 = wrapc(ax + 1, G.ncx, G.px);
            const int wy0 = wrapc(ay, G.ncy, G.py), wy1 = wrapc(ay + 1, G.ncy, G.py);
            const int cells = live ? nxs * nys : 0;
            double mx = 0.0, my = 0.0;
            int hits = 0;
            for (int ci = 0; ci < 4; ci++) {
                if (!__any_sync(full, ci < cells)) break;
                int q = 0, q1 = 0;
                if (ci < cells) {
                    const int cell = (ci / nxs ? wy1 : wy0) * G.ncx + (ci % nxs ? wx1 : wx0);
                    q = off[cell];
                    q1 = off[cell + 1];
                }
                for (; __any_sync(full, q < q1); q += 4) {
                    bool hit = false;
                    double px = 0.0, py = 0.0, push = 0.0;
                    bool apart = false;
                    if (q + sub < q1) {
                        const Cover e = cov[q + sub];
                        const double dx = pwrap(cx - e.x, G.Lx, G.px), dy = pwrap(cy - e.y, G.Ly, G.py);
                        const double d = sqrt(dx * dx + dy * dy);
                        const double sep = rad + e.r;
                        if (d < sep) {
                            int jax, jbx, jay, jby;
                            cell_span(e.x - e.r, e.x + e.r, G.cwx, G.ncx, G.px, jax, jbx);
                            cell_span(e.y - e.r, e.y + e.r, G.cwy, G.ncy, G.py, jay, jby);
                            bool seen = false;
                            for (int cj = 0; cj < ci && !seen; cj++)
                                seen = in_span(cj % nxs ? wx1 : wx0, jax, jbx, G.ncx, G.px) &&
                                       in_span(cj / nxs ? wy1 : wy0, jay, jby, G.ncy, G.py);
                            if (!seen) {
                                hit = true;
                                push = (sep - d) * 1.0001 + 1e-9 * sep;
                                apart = d > 0;
                                if (apart) { px = dx / d; py = dy / d; }
                            }
                        }
                    }
                    // the attempt's hits in order
                    const unsigned mine = __ballot_sync(full, hit) >> quad & 15u;
                    for (int k = 0; k < 4; k++) {
                        if (!__any_sync(full, mine >> k & 1u)) continue;
                        const double hx = __shfl_sync(full, px, k, 4), hy = __shfl_sync(full, py, k, 4);
                        const double hp = __shfl_sync(full, push, k, 4);
                        const bool ha = __shfl_sync(full, (int)apart, k, 4) != 0;
                        if (!(mine >> k & 1u)) continue;
                        if (ha) { mx += hx * hp; my += hy * hp; }
                        else mx += hp;
                        hits++;
                    }
                }
            }
            if (live && !hits) {
                found = true;
                live = false;
            }
            // attempts after a successful one stop
            const unsigned ok = __ballot_sync(full, found);
            if (ok && att > (__ffs(ok) - 1) >> 2) live = false;
            if (!__any_sync(full, live)) break;
            if (live) {
                cx += mx;
                cy += my;
                if (G.px) cx -= G.Lx * floor(cx / G.Lx);
                else cx = fmin(fmax(cx, xlo), xhi);
                if (G.py) cy -= G.Ly * floor(cy / G.Ly);
                else cy = fmin(fmax(cy, ylo), yhi);
            }
        }
        const unsigned ok = __ballot_sync(full, found);
        if (lane == (ok ? __ffs(ok) - 1 : 0)) {
            cand[i] = ok != 0;
            if (ok) {
                tx[i] = cx;
                ty[i] = cy;
            }
        }
    }
}

GD_DEV int cand_cell(const PGrid &G, double x, double y)
{
    const int cx = min(max((int)floor(x / G.cwx), 0), G.ncx - 1);
    const int cy = min(max((int)floor(y / G.cwy), 0), G.ncy - 1);
    return cy * G.ncx + cx;
}

// The free positions by cell (k_cover's two passes).
template <bool FILL>
__global__ void k_cands(int c0, int c1, const unsigned char *cand, const double *tx, const double *ty, PGrid G,
                        int *cnt, const int *off, int *list)
{
    for (int i = c0 + blockIdx.x * blockDim.x + threadIdx.x; i < c1; i += gridDim.x * blockDim.x) {
        if (!cand[i]) continue;
        const int c = cand_cell(G, tx[i], ty[i]);
        if (FILL) list[off[c] + atomicSub(&cnt[c], 1) - 1] = i;
        else atomicAdd(&cnt[c], 1);
    }
}

// Step 2: a free position is kept unless a free position of a lower-index
// disk of the class overlaps it (class radii are at most half a cell, so
// such a disk's centre lies in one of the 3 x 3 cells around).
__global__ void k_accept(int c0, int c1, const double *r, const unsigned char *cand, const double *tx,
                         const double *ty, PGrid G, const int *off, const int *list, unsigned char *placed, double *x,
                         double *y, int *nplaced)
{
    for (int i = c0 + blockIdx.x * blockDim.x + threadIdx.x; i < c1; i += gridDim.x * blockDim.x) {
        if (!cand[i]) continue;
        const int own = cand_cell(G, tx[i], ty[i]), cx = own % G.ncx, cy = own / G.ncx;
        bool ok = true;
        for (int dyc = -1; dyc <= 1 && ok; dyc++)
            for (int dxc = -1; dxc <= 1 && ok; dxc++) {
                int xx = cx + dxc, yy = cy + dyc;
                if (G.px) xx = wrapc(xx, G.ncx, 1); else if (xx < 0 || xx >= G.ncx) continue;
                if (G.py) yy = wrapc(yy, G.ncy, 1); else if (yy < 0 || yy >= G.ncy) continue;
                // small grids: a wrapped neighbour may repeat the own cell or
                // another; repeats only repeat the same tests
                const int cell = yy * G.ncx + xx;
                for (int q = off[cell]; q < off[cell + 1]; q++) {
                    const int j = list[q];
                    if (j >= i) continue;
                    const double dx = pwrap(tx[i] - tx[j], G.Lx, G.px), dy = pwrap(ty[i] - ty[j], G.Ly, G.py);
                    if (sqrt(dx * dx + dy * dy) < r[i] + r[j]) { ok = false; break; }
                }
            }
        if (ok) {
            placed[i] = 1;
            x[i] = tx[i];
            y[i] = ty[i];
            atomicAdd(nplaced, 1);
        }
    }
}

// One device allocation, cut into pieces of 256-byte alignment.
struct Arena {
    char *base = nullptr;
    size_t used = 0;
    ~Arena() { if (base) cudaFree(base); }
    template <class T> T *take(size_t count) {
        T *p = (T *)(base + used);
        used += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
};

int grid_n(long long n, int block) { return (int)std::max(1LL, std::min<long long>((n + block - 1) / block, 148LL * 16)); }

}  // namespace

// engine.cu: the thread's last error message
void set_last_error(const std::string &msg);

int place_disks(int n, const double *r_in, double Lx, double Ly, int px, int py, uint64_t seed, int max_rounds,
                double gap, double *x_out, double *y_out, int *placed_out)
{
    // largest first; ties keep input order
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return r_in[a] > r_in[b]; });
    std::vector<double> rs(n);
    for (int k = 0; k < n; k++) rs[k] = r_in[order[k]] + 0.5 * gap;
    const double rmin = std::max(rs[n - 1], 1e-9);
    auto cls = [&](double v) { return (int)std::floor(std::log2(std::max(v / rmin, 1.0))); };

    // the classes and their grids; the most cells of one and the most cells
    // the bounding boxes of all disks placed by its end can meet
    struct Class { int k0, k1, big; PGrid G; };
    std::vector<Class> classes;
    long long cells = 1, covers = 1;
    int widest = 1;
    for (int k0 = 0; k0 < n;) {
        // the class of disk k0: every disk down to half its class's radius
        Class C;
        C.k0 = k0;
        const int c = cls(rs[k0]);
        int k1 = k0;
        while (k1 < n && cls(rs[k1]) == c) k1++;
        C.k1 = k1;
        PGrid &G = C.G;
        G.Lx = Lx; G.Ly = Ly; G.px = px; G.py = py;
        const double cell = std::max(2.0 * rs[k0], 1e-9);
        G.ncx = std::max(1, std::min(8192, (int)std::floor(Lx / cell)));
        G.ncy = std::max(1, std::min(8192, (int)std::floor(Ly / cell)));
        G.cwx = Lx / G.ncx;
        G.cwy = Ly / G.ncy;
        double met = 0.0;
        C.big = 0;
        for (int k = 0; k < k1; k++) {
            const double own = cells_met(rs[k], G.cwx, G.ncx) * cells_met(rs[k], G.cwy, G.ncy);
            met += own;
            if (own > COVER_ALONE) C.big = k + 1;
        }
        if (met >= 2147483647.0) { set_last_error("too many cells covered"); return GODAR_ERR_NOMEM; }
        covers = std::max(covers, (long long)met);
        cells = std::max(cells, (long long)G.ncx * G.ncy);
        widest = std::max(widest, k1 - k0);
        classes.push_back(C);
        k0 = k1;
    }
    const size_t nc = (size_t)cells;
    const auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    Arena M;
    const size_t want = 5 * up((size_t)n * 8) + 2 * up((size_t)n) + 2 * up((nc + 1) * 4) + 2 * up(nc * 4) +
                        up((nc / 2048 + 64) * 4) + up((size_t)covers * 4) + up((size_t)covers * sizeof(Cover)) +
                        up((size_t)widest * 4) + up(16);
    cudaError_t got_mem = cudaMalloc(&M.base, want);
    if (got_mem == cudaErrorMemoryAllocation && release_kept()) {
        cudaGetLastError();
        got_mem = cudaMalloc(&M.base, want);
    }
    if (got_mem != cudaSuccess) {
        cudaGetLastError();
        M.base = nullptr;
        set_last_error("device allocation failed");
        return GODAR_ERR_NOMEM;
    }
    double *r = M.take<double>(n), *x = M.take<double>(n), *y = M.take<double>(n);
    double *tx = M.take<double>(n), *ty = M.take<double>(n);
    unsigned char *placed = M.take<unsigned char>(n), *cand = M.take<unsigned char>(n);
    // per cell: places in the lists of placed disks and of free positions, and
    // the counts they come from (zero between uses: the second pass of each
    // list counts them down)
    int *off = M.take<int>(nc + 1), *off2 = M.take<int>(nc + 1), *cnt = M.take<int>(nc), *cnt2 = M.take<int>(nc);
    int *scr = M.take<int>(nc / 2048 + 64);
    int *list = M.take<int>((size_t)covers);
    Cover *cov = M.take<Cover>((size_t)covers);
    int *list2 = M.take<int>(widest), *counter = M.take<int>(4);
    cudaMemcpy(r, rs.data(), (size_t)n * 8, cudaMemcpyHostToDevice);
    cudaMemset(placed, 0, (size_t)n);
    cudaMemset(cnt, 0, nc * 4);
    cudaMemset(cnt2, 0, nc * 4);
    cudaMemset(counter, 0, 16);
    int total_placed = 0;
    for (const Class &C : classes) {
        const PGrid G = C.G;
        const int k0 = C.k0, k1 = C.k1, m = k1 - k0, ncell = G.ncx * G.ncy;
        int left = m;
        for (int round = 0; round < max_rounds && left > 0; round++) {
            // coverage of every disk placed so far (they come before k1)
            k_cover<false><<<grid_n(C.big ? 1 << 20 : k1, 256), 256>>>(k1, C.big, x, y, r, placed, G, cnt, nullptr, nullptr);
            scan_excl(cnt, off, ncell, scr, 0);
            k_cover<true><<<grid_n(C.big ? 1 << 20 : k1, 256), 256>>>(k1, C.big, x, y, r, placed, G, cnt, off, list);
            k_cover_order<<<grid_n(ncell, 128), 128>>>(ncell, off, list, x, y, r, cov);
            // step 1
            k_trial<<<grid_n((long long)m * 32, 256), 256>>>(k0, k1, r, placed, G, off, cov, seed, round, cand, tx, ty);
            // step 2
            k_cands<false><<<grid_n(m, 256), 256>>>(k0, k1, cand, tx, ty, G, cnt2, nullptr, nullptr);
            scan_excl(cnt2, off2, ncell, scr, 0);
            k_cands<true><<<grid_n(m, 256), 256>>>(k0, k1, cand, tx, ty, G, cnt2, off2, list2);
            k_accept<<<grid_n(m, 128), 128>>>(k0, k1, r, cand, tx, ty, G, off2, list2, placed, x, y, counter);
            int got = 0;
            if (cudaMemcpy(&got, counter, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
                set_last_error("placement kernels failed");
                return GODAR_ERR_CUDA;
            }
            left -= got - total_placed;
            total_placed = got;
        }
        if (left > 0) break;     // the caller enlarges the domain
    }
    std::vector<double> hx(n), hy(n);
    std::vector<unsigned char> hp(n);
    cudaMemcpy(hx.data(), x, (size_t)n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(hy.data(), y, (size_t)n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(hp.data(), placed, (size_t)n, cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess) {
        set_last_error("placement kernels failed");
        return GODAR_ERR_CUDA;
    }
    for (int k = 0; k < n; k++) {
        x_out[order[k]] = hp[k] ? hx[k] : NAN;
        y_out[order[k]] = hp[k] ? hy[k] : NAN;
    }
    if (placed_out) *placed_out = total_placed;
    return GODAR_OK;
}

}  // namespace godar

extern "C" int godar_gpu_place(int n, const double *r, double Lx, double Ly, int periodic_x, int periodic_y,
                               uint64_t seed, int max_rounds, double gap, double *x, double *y, int *placed)
{
    if (n <= 0 || !r || !x || !y || !(Lx > 0) || !(Ly > 0) || !std::isfinite(Lx) || !std::isfinite(Ly) ||
        max_rounds <= 0 || !std::isfinite(gap))
        return GODAR_ERR_BAD_INPUT;
    // a negative gap lets disks overlap by up to -gap, as long as every
    // disk keeps a positive placement radius r + gap / 2
    for (int i = 0; i < n; i++)
        if (!(r[i] > 0) || !std::isfinite(r[i]) || !(r[i] + 0.5 * gap > 0)) return GODAR_ERR_BAD_INPUT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return GODAR_ERR_NO_DEVICE;
    }
    return godar::place_disks(n, r, Lx, Ly, periodic_x != 0, periodic_y != 0, seed, max_rounds, gap, x, y, placed);
}
