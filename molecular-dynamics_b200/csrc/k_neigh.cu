// k_neigh.cu -- reneighbour kernels of the tinyMD B200 timestep:
//   * periodic wrap of locals        (core/compute.impala:118-122, comm/comm.impala:152-162)
//   * ghost generation (borders)     (comm/comm.impala:105-127, 528-642, 723-734; comm/lb.impala:88-100)
//   * cell binning as a counting sort that reorders the device arrays by cell
//                                    (core/grid.impala:280-321, 406-426)
//   * neighbour-list build (core/neighborlist.impala:1-78): a block per cell,
//     the stencil's candidates filtered by the homes' bounding box and staged
//     in shared memory, a warp testing 32 of them against a home at once; or
//     eight lanes per home where cells hold few atoms or most hold none
//
// Ghost order.  The reference runs six passes (x+, x-, y+, y-, z+, z-); a
// pass scans locals then all earlier ghosts in order and appends the ones
// within one cell of the face, shifted by one box length.  A ghost is
// therefore identified by its root local r and its pass combination
// (ex, ey, ez) with e in {0 none, 1 plus pass, 2 minus pass}, and the
// reference appends them grouped by base-3 type index ez*9 + ey*3 + ex - 1,
// in increasing r inside a type.  The kernels below compute that order
// directly: one mask per local, per-type counts, one exclusive scan, emit.
//
// In-cell order.  The reference fills cells sequentially by particle index,
// so a cell lists its locals in input order, then its ghosts in ghost order.
// The counting sort here ranks each cell's members by that reference index,
// which makes list order -- and hence FP64 force summation order -- equal to
// the reference's.

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdio>

#include "comm.h"
#include "md_common.cuh"
#include "launch.cuh"
#include "md_state.h"

namespace tmd {

namespace {

struct GeoArgs {
    double wlo[3], whi[3], alo[3], ahi[3], len[3];
    double spacing;
    int nx, ny, nz, ncells;
    double rb_h, inv_rb_h;
};

GeoArgs geo_args(const Geometry& g) {
    GeoArgs a;
    for (int d = 0; d < 3; ++d) {
        a.wlo[d] = g.world_lo[d];
        a.whi[d] = g.world_hi[d];
        a.alo[d] = g.aabb_lo[d];
        a.ahi[d] = g.aabb_hi[d];
        a.len[d] = g.len[d];
    }
    a.spacing = g.spacing;
    a.nx = g.nx;
    a.ny = g.ny;
    a.nz = g.nz;
    a.ncells = g.ncells;
    a.rb_h = g.rb_h;
    a.inv_rb_h = 1.0 / g.rb_h;
    return a;
}

__device__ __forceinline__ double comp(const double4& p, int d) { return d == 0 ? p.x : (d == 1 ? p.y : p.z); }

// core/grid.impala:406-411 and 419-426: floor per axis, flattened, with only
// the global range check.  Returns ncells when outside.
__device__ __forceinline__ int flat_cell(const double4& p, const GeoArgs& a) {
    int i = (int)floor(ddiv(dsub(p.x, a.alo[0]), a.spacing));
    int j = (int)floor(ddiv(dsub(p.y, a.alo[1]), a.spacing));
    int k = (int)floor(ddiv(dsub(p.z, a.alo[2]), a.spacing));
    int c = (k * a.ny + j) * a.nx + i;
    return (c >= 0 && c < a.ncells) ? c : a.ncells;
}

// The rebasing cell is computed here only (the binning's move) and stored, so every kernel sees
// the same cell; a product with 1 / h instead of a correctly rounded division is enough (a pair
// within the list cutoff stays within one cell step whatever the rounding at a cell boundary).
__device__ __forceinline__ int rebase_cell(const double4& p, const GeoArgs& a) {
    int i = (int)floor((p.x - a.alo[0]) * a.inv_rb_h);
    int j = (int)floor((p.y - a.alo[1]) * a.inv_rb_h);
    int k = (int)floor((p.z - a.alo[2]) * a.inv_rb_h);
    return pack3(i, j, k);
}

}  // namespace

// ---- periodic wrap ---------------------------------------------------------
// comm/comm.impala:152-162: one wrap per axis with strict comparisons against
// the world box.  img counts wraps so the adjoint can unwrap displacements.
__device__ __forceinline__ double4 wrap_local(double4* __restrict__ pos, int* __restrict__ img, int i,
                                              const GeoArgs& a) {
    double4 p = ld_d4(pos + i);
    double c[3] = {p.x, p.y, p.z};
    int im = img[i];
    int w[3] = {unpack_axis(im, 0), unpack_axis(im, 1), unpack_axis(im, 2)};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double v = comp(p, d);
        if (v < a.wlo[d]) { c[d] = dadd(c[d], a.len[d]); w[d] -= 1; }
        if (v > a.whi[d]) { c[d] = dsub(c[d], a.len[d]); w[d] += 1; }
    }
    p = make_double4(c[0], c[1], c[2], p.w);
    st_d4(pos + i, p);
    img[i] = pack3(w[0], w[1], w[2]);
    return p;
}

__global__ void k_enforce_pbc(double4* __restrict__ pos, int* __restrict__ img, int N, GeoArgs a) {
    const int blk = (int)blockIdx.x + pdl_wait();
    int i = blk * blockDim.x + threadIdx.x;
    if (i >= N) return;
    wrap_local(pos, img, i, a);
}

// ---- borders ---------------------------------------------------------------
// Mask of the 26 ghost types of one local (bit t = ez*9 + ey*3 + ex - 1) in
// bits 0-25 and the six periodic flags of its passes in bits 26-31
// (x+, x-, y+, y-, z+, z-): flag set means the pass shifts that axis.
__device__ __forceinline__ unsigned border_mask(const double4& p, const GeoArgs& a) {
    const double dsp = dmul(a.spacing, 2.0);
    unsigned has[3] = {0, 0, 0};  // bit0 plus pass, bit1 minus pass
    unsigned flags = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double v = comp(p, d);
        // comm/comm.impala:116-127 (grid.aabb is the extended rank box)
        if (v > dsub(a.ahi[d], dsp)) has[d] |= 1u;
        if (v < dadd(a.alo[d], dsp)) has[d] |= 2u;
        // comm/lb.impala:88-100 with the pass direction
        if (v > dsub(a.whi[d], a.spacing)) flags |= 1u << (2 * d);
        if (v < dadd(a.wlo[d], a.spacing)) flags |= 1u << (2 * d + 1);
    }
    unsigned mask = 0;
    for (int ez = 0; ez < 3; ++ez) {
        if (ez && !(has[2] & (1u << (ez - 1)))) continue;
        for (int ey = 0; ey < 3; ++ey) {
            if (ey && !(has[1] & (1u << (ey - 1)))) continue;
            for (int ex = 0; ex < 3; ++ex) {
                if (ex && !(has[0] & (1u << (ex - 1)))) continue;
                int t = ez * 9 + ey * 3 + ex;
                if (t) mask |= 1u << (t - 1);
            }
        }
    }
    return mask | (flags << 26);
}

// Pass 1: masks in reference order and per-block per-type counts [26][nblk].  WRAP: the
// periodic wrap of each local (k_enforce_pbc's) is done here first, one launch fewer.
template <bool WRAP>
__global__ void __launch_bounds__(kBorderThreads) k_border_count(double4* __restrict__ pos, int* __restrict__ img, const int* __restrict__ slot_of_ref,
                               unsigned* __restrict__ bmask, int* __restrict__ bcount, int N, int nblk, GeoArgs a,
                               int* __restrict__ cnt, int nseg, DevStatus* st) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ int wc[kBorderThreads / 32][26];
    const int r = blk * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // the binning that follows starts from zeroed cell counters and status (no memsets there)
    for (int g = r; g < nseg; g += gridDim.x * blockDim.x) cnt[g] = 0;
    if (r == 0) st->out_local = st->out_ghost = st->nchain = st->img_over1 = st->img_over2 = st->filled = 0;
    unsigned m = 0;
    if (r < N) {
        const int sl = slot_of_ref[r];
        m = border_mask(WRAP ? wrap_local(pos, img, sl, a) : ld_d4(pos + sl), a);
        bmask[r] = m;
    }
    for (int t = 0; t < 26; ++t) {
        unsigned b = __ballot_sync(0xffffffffu, (m >> t) & 1u);
        if (lane == 0) wc[wid][t] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x < 26) {
        int s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += wc[w][threadIdx.x];
        bcount[threadIdx.x * nblk + blk] = s;
    }
}

// Pass 2 (after an exclusive scan of bcount into boff): writes every ghost at
// slot N + g, g its reference ghost index, with its source / root links.
// MR (several ranks): only the types in selfmask are periodic ghosts of this rank; the others
// are images for the neighbour ranks, listed (root, type) in type order for the halo pack.
// tab[t] / tab[26 + t]: images of the other kind before type t (k_halo.cu's table).
struct RemoteOut {
    const int* tab;
    int* send_ref;
    int* send_type;
    unsigned selfmask;
};

template <bool MR>
__global__ void __launch_bounds__(kBorderThreads) k_border_emit(double4* __restrict__ pos, double4* __restrict__ vel, double4* __restrict__ frc,
                              double* __restrict__ mass, int* __restrict__ ref, int* __restrict__ slot_of_ref,
                              const unsigned* __restrict__ bmask, const int* __restrict__ boff,
                              int* __restrict__ gsrc, int* __restrict__ groot, int* __restrict__ gcode,
                              int* __restrict__ bsrc_ref, int* __restrict__ broot_ref, int* __restrict__ bcode,
                              int N, int nblk, int capA, GeoArgs a, int sync_vel, RemoteOut ro,
                              int* count_host) {
    const int blk = (int)blockIdx.x + pdl_wait();
    if (count_host && blk == 0 && threadIdx.x == 0)  // the ghost count, to the host that polls for it
        *reinterpret_cast<volatile int*>(count_host) = boff[26 * nblk];
    __shared__ int wpre[kBorderThreads / 32][26];
    __shared__ unsigned char s_rank[26][kBorderThreads];  // a thread's rank among its warp's ghosts of each type
    const int r = blk * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned m = r < N ? bmask[r] : 0u;
    const unsigned lt = lanemask_lt();
    for (int t = 0; t < 26; ++t) {
        unsigned b = __ballot_sync(0xffffffffu, (m >> t) & 1u);
        s_rank[t][threadIdx.x] = (unsigned char)__popc(b & lt);
        if (lane == 0) wpre[wid][t] = __popc(b);
    }
    __syncthreads();
    if (threadIdx.x < 26) {  // exclusive prefix over warps, per type
        int s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            int c = wpre[w][threadIdx.x];
            wpre[w][threadIdx.x] = s;
            s += c;
        }
    }
    __syncthreads();
    if (r >= N || (m & 0x03ffffffu) == 0) return;
    const int s_root = slot_of_ref[r];
    const double4 p = ld_d4(pos + s_root);
    const double mroot = mass[s_root];
    const double4 vroot = ld_d4(vel + s_root);
    const unsigned flags = m >> 26;
    // index of this root's ghost of type t (a type whose bit is set)
    auto gidx = [&](int t) { return boff[t * nblk + blk] + wpre[wid][t] + s_rank[t][threadIdx.x]; };
    for (int t = 0; t < 26; ++t) {
        if (!((m >> t) & 1u)) continue;
        if (MR && !((ro.selfmask >> t) & 1u)) {
            const int k = gidx(t) - ro.tab[26 + t];
            ro.send_ref[k] = r;
            ro.send_type[k] = t;
            continue;
        }
        const int g = gidx(t) - (MR ? ro.tab[t] : 0);
        const int slot = N + g;
        if (slot >= capA) continue;  // the host grows the arrays and redoes the pass
        const int tt = t + 1;
        const int e[3] = {tt % 3, (tt / 3) % 3, tt / 9};
        int last = e[2] ? 2 : (e[1] ? 1 : 0);
        double c[3] = {p.x, p.y, p.z};
        int tot[3] = {0, 0, 0};
        int lastsh = 0;
        for (int d = 0; d < 3; ++d) {
            if (!e[d]) continue;
            // plus pass shifts by -1 when the flag holds, minus pass by +1
            int sh = 0;
            if (e[d] == 1 && (flags & (1u << (2 * d)))) sh = -1;
            if (e[d] == 2 && (flags & (1u << (2 * d + 1)))) sh = 1;
            c[d] = dadd(c[d], dmul(a.len[d], (double)sh));
            tot[d] = sh;
            if (d == last) lastsh = sh;
        }
        // source of the last pass: the ghost of the same root without the last axis, or the root
        const int tsrc = tt - e[last] * (last == 0 ? 1 : (last == 1 ? 3 : 9));
        const int src_ref = tsrc == 0 ? r : N + gidx(tsrc - 1) - (MR ? ro.tab[tsrc - 1] : 0);
        const int src_slot = tsrc == 0 ? s_root : src_ref;  // a ghost's slot is its reference index
        int code = 0;
        for (int d = 0; d < 3; ++d) {
            int ls = (d == last) ? lastsh : 0;
            code |= (ls + 1) << (2 * d);
            code |= (tot[d] + 1) << (8 + 2 * d);
        }
        st_d4(pos + slot, make_double4(c[0], c[1], c[2], 0.0));
        mass[slot] = mroot;
        st_d4(frc + slot, make_double4(0.0, 0.0, 0.0, 0.0));
        st_d4(vel + slot, sync_vel ? vroot : make_double4(0.0, 0.0, 0.0, 0.0));
        ref[slot] = slot;
        slot_of_ref[slot] = slot;
        gsrc[g] = src_slot;
        groot[g] = s_root;
        gcode[g] = code;
        bsrc_ref[g] = src_ref;
        broot_ref[g] = r;
        bcode[g] = code;
    }
}

// ---- binning (counting sort) -----------------------------------------------
// cnt / cstart layout: [0, ncells] locals per cell (index ncells = outside
// the grid), [ncells+1, 2*ncells+1] ghosts per cell.
__global__ void k_bin_count(const double4* __restrict__ pos, int* __restrict__ cnt, int* __restrict__ bin_cell,
                            int* __restrict__ bin_rank, DevStatus* st, int N, int NA, GeoArgs a) {
    const int blk = (int)blockIdx.x + pdl_wait();
    int s = blk * blockDim.x + threadIdx.x;
    if (s >= NA) return;
    int c = flat_cell(ldg_d4(pos + s), a);
    if (c == a.ncells) atomicAdd(s < N ? &st->out_local : &st->out_ghost, 1);
    int seg = s < N ? c : (a.ncells + 1) + c;
    bin_cell[s] = c;
    bin_rank[s] = atomicAdd(&cnt[seg], 1);
}

__global__ void k_bin_scatter(const int* __restrict__ ref, const int* __restrict__ bin_cell,
                              const int* __restrict__ bin_rank, const int* __restrict__ cstart,
                              int* __restrict__ tmp_key, int* __restrict__ tmp_src, int N, int NA, int ncells) {
    const int blk = (int)blockIdx.x + pdl_wait();
    int s = blk * blockDim.x + threadIdx.x;
    if (s >= NA) return;
    int c = bin_cell[s];
    int seg = s < N ? c : (ncells + 1) + c;
    int p = cstart[seg] + bin_rank[s];
    tmp_key[p] = ref[s];
    tmp_src[p] = s;
}

// The members of a segment (a cell's locals or its ghosts) ranked by reference index (keys are
// unique), each moved from its old slot to its new one (cstart[segment] + rank).  The two
// outside-the-grid buckets keep arrival order: their members have no neighbours and are
// nobody's neighbour, so their order is not observable.
struct MoveArgs {
    const double4* pos_o; double4* pos_n;
    const double4* vel_o; double4* vel_n;
    const double4* frc_o; double4* frc_n;
    const double* mass_o; double* mass_n;
    const int* ref_o; int* ref_n;
    const int* img_o; int* img_n;
    int* slot_of_ref; int* rref; int* rbk;
    const int* bin_cell; int* slot_cell;
    float4* pos32; int* img_cnt; int* img_slot;
    int capA, N, mixed;
};

__device__ __forceinline__ void move_slot(int n, int o, const MoveArgs& m, const GeoArgs& a) {
    m.slot_cell[n] = m.bin_cell[o];
    const double4 p = ldg_d4(m.pos_o + o);
    const double4 v = ldg_d4(m.vel_o + o), f = ldg_d4(m.frc_o + o);
    st_d4(m.pos_n + n, p);
    st_d4(m.vel_n + n, v);
    st_d4(m.frc_n + n, f);
    m.mass_n[n] = m.mass_o[o];
    const int r = m.ref_o[o];
    m.ref_n[n] = r;
    if (n < m.N) {
        m.img_n[n] = m.img_o[o];
        m.rref[n] = r;
        // empty image records for k_ghost_links to fill
        m.img_cnt[n] = 0;
        m.img_cnt[m.capA + n] = 0;
#pragma unroll
        for (int k = 0; k < kImgW; ++k) m.img_slot[(size_t)k * m.capA + n] = -1;
    }
    m.slot_of_ref[r] = n;
    const int k = rebase_cell(p, a);
    m.rbk[n] = k;
    if (m.mixed) m.pos32[n] = rebased32(p, k, a.alo, a.rb_h);
}

// One thread per new slot: the slot's segment (cell, locals or ghosts) from its old slot's cell,
// its rank among the segment's members by reference index, then the move.  (A warp per segment
// left ~45 % of the lanes idle and half the warps on the empty ghost segments of inner cells.)
__global__ void k_rank_move(const int* __restrict__ cstart, const int* __restrict__ tmp_key,
                            const int* __restrict__ tmp_src, int NA, int ncells, MoveArgs m, GeoArgs ga,
                            DevStatus* st) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int e = blk * blockDim.x + threadIdx.x;
    // the list build that follows starts from a zeroed status (no memset there)
    if (e == 0) st->max_nb = 0;
    const int o = e < NA ? tmp_src[e] : 0;
    const int key = e < NA ? tmp_key[e] : 0;
    const int c = e < NA ? m.bin_cell[o] : ncells;
    int n = e;  // atoms outside the grid keep their bucket order
    bool first = false;
    if (c != ncells) {
        const int seg = o < m.N ? c : ncells + 1 + c;
        const int a = cstart[seg], b = cstart[seg + 1];
        int rank = 0;
        for (int f = a; f < b; ++f) rank += tmp_key[f] < key;
        n = a + rank;
        first = rank == 0 && o < m.N;
    }
    // cells that hold locals (the next list build's choice of kernel)
    const int filled = __syncthreads_count(first);
    if (threadIdx.x == 0 && filled) atomicAdd(&st->filled, filled);
    if (e >= NA) return;
    move_slot(n, o, m, ga);
}

// Per ghost: its source, root and shift code in slot terms, and its place in the image
// records of the locals (k_rank_move emptied them): a local's direct two-phase images (ghosts
// whose source it is) and all its images (ghosts whose root it is), one plane per image
// number (filled in order, -1 beyond the last); ghosts whose two-phase source is another
// ghost go to `chain`.  The order within a record follows the atomics, but every ghost is
// written exactly once, so the result is deterministic.
struct LinkArgs {
    const int* ref; const int* slot_of_ref; const int* bsrc_ref; const int* broot_ref; const int* bcode;
    int* gsrc; int* groot; int* gcode; int* rref; int* img_cnt; int* img_slot; int* chain;
    DevStatus* st;
    int N, G, capA;
};

__device__ __forceinline__ void ghost_link(int h, const LinkArgs& l) {
    const int N = l.N, capA = l.capA;
    int g = l.ref[N + h] - N;
    if (l.broot_ref[g] < 0) {  // received from another rank: refreshed by the halo exchange
        l.gsrc[h] = l.groot[h] = -1;
        l.gcode[h] = 0;
        l.rref[N + h] = -1;
        return;
    }
    const int s1 = l.slot_of_ref[l.bsrc_ref[g]];
    const int r = l.slot_of_ref[l.broot_ref[g]];
    l.gsrc[h] = s1;
    l.groot[h] = r;
    l.gcode[h] = l.bcode[g];
    l.rref[N + h] = l.broot_ref[g];
    const int t = N + h;
    if (s1 < N) {
        const int k = atomicAdd(&l.img_cnt[s1], 1);
        if (k < kImg1) l.img_slot[(size_t)k * capA + s1] = t;
        else atomicAdd(&l.st->img_over1, 1);
    } else {
        l.chain[atomicAdd(&l.st->nchain, 1)] = h;
    }
    const int k2 = atomicAdd(&l.img_cnt[capA + r], 1);
    if (k2 < kImg2) l.img_slot[(size_t)(kImg1 + k2) * capA + r] = t;
    else atomicAdd(&l.st->img_over2, 1);
}

__global__ void k_ghost_links(LinkArgs l) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int h = blk * blockDim.x + threadIdx.x;
    if (h < l.G) ghost_link(h, l);
}

// ---- neighbour lists ---------------------------------------------------------
// rebasing cell k relative to b as dx + 4 dy + 16 dz (signed offsets per axis): for two atoms
// whose offsets differ by at most 1 on every axis, (c - i) + 21 is exactly the list code
// (dx+1) | (dy+1) << 2 | (dz+1) << 4 of the pair, each term being 0, 1 or 2 with no carry
__device__ __forceinline__ int rel_code(int k, int b) {
    return wrap_diff(unpack_axis(k, 0), unpack_axis(b, 0)) + 4 * wrap_diff(unpack_axis(k, 1), unpack_axis(b, 1)) +
           16 * wrap_diff(unpack_axis(k, 2), unpack_axis(b, 2));
}
constexpr int kCodeBias = 1 + 4 + 16;  // dk + 1 on every axis

// The reference's exact FP64 membership test for a pair near the list cutoff (core/neighborlist.impala:
// 18-78), which the FP32 prefilter cannot decide (~1 candidate in 150)
__device__ __forceinline__ bool exact_within(const double4* __restrict__ pos, int i, int j, double cut2) {
    const double4 pi = pos[i], pj = pos[j];
    return len2_strict(dsub(pi.x, pj.x), dsub(pi.y, pj.y), dsub(pi.z, pj.z)) <= cut2;
}

// A block builds the lists of one cell's atoms, the homes, 32 at a time (core/neighborlist.impala:
// 18-78).  The 27 stencil cells' atoms (locals then ghosts per cell, in stencil order) are staged in
// shared memory in order, keeping those within the list cutoff (plus the FP32 margin) of the homes'
// bounding box; then each warp takes every fourth home and tests 32 staged candidates at once, one
// per lane.  The ballot of the hits gives each hit its place, so a list comes out in stencil order --
// the reference's, which fixes the FP64 summation order.  A home's entries collect in shared memory
// and leave as whole quads.  Pairs near the cutoff take the reference's FP64 test (rsq <= cutoff^2),
// so membership is exactly the reference's; the FP32 margin follows from the magnitude of the staged
// coordinates (margin32), which makes that test rare.
//
// Bound by instruction issue (77 %): 67 M warp instructions at 131,072 atoms, 46 M of them the pair
// tests, 16 M the staging, 5 M the blocks' start; without the tests the kernel takes 36 of 85 us, without
// the staging too 18 us (the chain of loads and barriers that starts a block).  One warp per cell with a home per lane walking the
// candidates one by one, as this kernel did before, took 83 M (19 of 32 lanes held a home) and made
// small systems wait for one serial walk.  Measured before -> now (us): 256 atoms 43 -> 15, 2,048
// 48 -> 18, 16,384 51 -> 23, 131,072 124 -> 91, 442,368 336 -> 268; half lists at 131,072 167 -> 102
// (105 where they hold their local pairs from both sides).  More blocks per SM: 98-104 us at 131,072 with 9, 10
// or 12 (56, 48, 40 registers: spills).
// A step of 1, 3 or 4 chunks instead of 2: 97, 92, 96 us at 131,072; the FP64 test or the emptying of
// a full buffer inside the step loop, where the compiler predicates it: 130 us.
//
// List layout: quads of four consecutive entries of one atom, atom-fastest (nl_index): a force
// kernel reads four entries with one 16-byte load, and the quads of a warp's 32 atoms form one
// 512-byte line.  An entry is slot << 6 | code, code = dk + 1 per axis, dk the neighbour's
// rebasing cell minus the home's (mixed form).  A list's last quad is padded with the home
// itself one rebasing cell away on every axis (code 42), which every force kernel skips by
// count or finds beyond its cutoff.
constexpr int kNlThreads = 128, kNlWarps = kNlThreads / 32;
constexpr int kNlChunks = 5;                // candidates staged per lane and tile
constexpr int kNlTile = kNlThreads * kNlChunks;  // candidates staged at once
constexpr int kNlStep = 2;                  // chunks of 32 candidates a home tests at once
constexpr int kNlBuf = 128 + 32 * kNlStep;  // entries of a home collected before they leave as quads
constexpr uint32_t kPadCode = 42u;          // dk = +1 on every axis

struct NlArgs {
    double cut2;  // cutoff^2 (FP64, the reference's membership test)
    float cut;
    float wide2;  // an FP32 window that reaches it may hold pairs of |dk| > 1 (far_homes)
    int nbcap, stride, N, ncells, nx, nxy;
    int two;  // half lists: local pairs from both sides (two_sided)
    double alo[3], spacing;
};

// Bound of |r^2 (FP32) - r^2 (exact)| for a pair near the cutoff whose staged coordinates are at
// most `mag` in magnitude: each coordinate is rounded once (2^-24 mag) and so is each difference
// (2^-24 cut), an error of del below 3 * 2^-24 mag per axis, of r^2 below 2 sqrt(3) cut times that
// plus 3 roundings of r^2; three times that sum is taken.
__device__ __forceinline__ float margin32(float cut, float mag) {
    constexpr float u = 1.0f / 16777216.0f;
    return 3.0f * (10.4f * u * cut * fmaxf(mag, cut) + 3.0f * u * cut * cut);
}

__device__ __forceinline__ float warp_min(float v) {
    asm("redux.sync.min.f32 %0, %0, 0xffffffff;" : "+f"(v));
    return v;
}

// shared memory by its 32-bit address (the walk's inner loop steps addresses, not indices)
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 lds_f4(uint32_t p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p));
    return v;
}
__device__ __forceinline__ int lds_i(uint32_t p) {
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ void sts_u(uint32_t p, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
}

// writes the quads of buf[0, n) (n a multiple of four) to the list of atom i from entry k0 on
__device__ __forceinline__ void store_quads(const uint32_t* buf, int n, int k0, int i, uint32_t* __restrict__ nbl,
                                            const NlArgs& a, int lane) {
    for (int q = lane; 4 * q < n; q += 32)
        if (k0 + 4 * q < a.nbcap)
            reinterpret_cast<uint4*>(nbl)[(size_t)((k0 >> 2) + q) * a.stride + i] =
                reinterpret_cast<const uint4*>(buf)[q];
}

// the buffer holds 128 entries or more: 32 whole quads leave and the rest moves up; a later tile's
// list that starts inside a quad leaves entry by entry
__device__ __forceinline__ void drain(uint32_t* buf, int& nb, int& out, int i, uint32_t* __restrict__ nbl,
                                   const NlArgs& a, int lane) {
    __syncwarp();
    if ((out & 3) == 0) {
        store_quads(buf, 128, out, i, nbl, a, lane);
        nb -= 128;
        out += 128;
        uint32_t rest[kNlStep];
#pragma unroll
        for (int u = 0; u < kNlStep; ++u) rest[u] = buf[128 + 32 * u + lane];
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kNlStep; ++u)
            if (32 * u + lane < nb) buf[32 * u + lane] = rest[u];
    } else {
        for (int e = lane; e < nb; e += 32)
            if (out + e < a.nbcap) nbl[nl_index(out + e, i, a.stride)] = buf[e];
        out += nb;
        nb = 0;
        __syncwarp();
    }
}

// The lists of homes hb .. hb + hn - 1, one of them far outside the cell: the binning tests only the
// flattened cell index, so a coordinate may be anything, infinite too.  The FP32 margin grows with it,
// and past wide2 the window takes in pairs of |dk| > 1, whose entries do not give back the candidate's
// slot.  Every candidate takes the FP64 test here (rare: out of line, so that the walk keeps its registers).
// both: local candidates below it always pass a half list's reference test (two-sided lists).
template <int HM>
__device__ __noinline__ int far_homes(const double4* __restrict__ pos, const int* __restrict__ ref,
                                      const int* __restrict__ rbk, int* __restrict__ nbn,
                                      uint32_t* __restrict__ nbl, double cut2, int nbcap, int stride, int both,
                                      int hb, int hn, int nr, const int* rstart, const int* rpre) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    int most = 0;
    for (int i = hb + (int)(threadIdx.x >> 5); i < hb + hn; i += kNlWarps) {
        const int rb = __ldg(rbk + i), iref = HM ? __ldg(ref + i) : 0, M = rpre[nr];
        int cnt = 0, r = 0;
        for (int m0 = 0; m0 < M; m0 += 32) {
            const int m = m0 + lane;
            while (m < M && rpre[r + 1] <= m) ++r;
            const int slot = m < M ? rstart[r] + m - rpre[r] : i;
            const bool may = slot != i && (!HM || slot < both || __ldg(ref + slot) < iref);
            const bool take = may && exact_within(pos, i, slot, cut2);
            const unsigned hits = __ballot_sync(0xffffffffu, take);
            const int k = cnt + __popc(hits & lt);
            if (take && k < nbcap)
                nbl[nl_index(k, i, stride)] =
                    ((uint32_t)slot << kCodeBits) + (uint32_t)(rel_code(__ldg(rbk + slot), rb) + kCodeBias);
            cnt += __popc(hits);
        }
        if (lane < ((-cnt) & 3) && cnt + lane < nbcap)  // the last quad's padding
            nbl[nl_index(cnt + lane, i, stride)] = ((uint32_t)i << kCodeBits) | kPadCode;
        if (lane == 0) nbn[i] = cnt;
        most = max(most, cnt);
    }
    return most;
}

template <int HM>
__global__ void __launch_bounds__(kNlThreads, 8)
k_build_list(const double4* __restrict__ pos, const int* __restrict__ ref, const int* __restrict__ rbk,
             const int* __restrict__ cstart, int* __restrict__ nbn, uint32_t* __restrict__ nbl, DevStatus* st,
             NlArgs a, int cell_blocks, LinkArgs la) {
    const int blk = (int)blockIdx.x + pdl_wait();
    // candidate position (cell-centre relative); w = slot << 6 + its rebasing cell relative to the
    // first home's (rel_code) + kCodeBias, from which a home's entry is one subtraction
    __shared__ float4 s_cand[kNlTile + 32 * kNlStep];
    __shared__ int s_cref[HM ? kNlTile + 32 * kNlStep : 1];
    __shared__ float4 s_home[32];  // position; w = its relative rebasing cell
    __shared__ int s_href[HM ? 32 : 1];
    __shared__ int s_cnt[32];      // entries of each home so far (cells of more than one tile)
    __shared__ int s_rstart[54];   // the stencil's ranges: first slot, candidates before it
    __shared__ int s_rpre[55];
    __shared__ int s_nr;
    __shared__ int s_slot[kNlTile];  // slots of the tile's candidates
    __shared__ float4 s_box[2];    // the homes' bounding box; w = r^2 certainly inside, outside
    __shared__ double s_ctr[3];    // the cell's centre
    __shared__ int s_rb0;          // the first home's rebasing cell
    __shared__ int s_kept[kNlWarps];
    __shared__ __align__(16) uint32_t s_buf[kNlThreads / 32][kNlBuf];

    if (blk >= cell_blocks) {  // blocks past the cells link the ghosts (k_ghost_links' work)
        const int h = (blk - cell_blocks) * blockDim.x + threadIdx.x;
        if (h < la.G) ghost_link(h, la);
        return;
    }
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blk;
    const int h0 = cstart[c], h1 = cstart[c + 1];
    if (h0 == h1) return;
    const unsigned lt = lanemask_lt();

    // 27 stencil cells in the reference order (z, y, x offsets -1..1), each contributing its locals
    // then its ghosts: 54 ranges of slots.  Without ghosts around, the three cells of an x row are one
    // range: 9 ranges.  One warp of the group finds them while another looks at the homes.
    if (wid == 0) {
        int start = 0, len = 0, gs = 0, gl = 0;
        if (lane < 27) {
            const int oz = lane / 9 - 1, oy = (lane / 3) % 3 - 1, ox = lane % 3 - 1;
            const int nb = c + oz * a.nxy + oy * a.nx + ox;
            if (nb >= 0 && nb < a.ncells) {
                start = cstart[nb];
                len = cstart[nb + 1] - start;
                gs = cstart[a.ncells + 1 + nb];
                gl = cstart[a.ncells + 2 + nb] - gs;
            }
        }
        const bool ghosts = __any_sync(0xffffffffu, gl > 0);
        int incl = len + gl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int ex = incl - len - gl;
        if (ghosts) {
            if (lane < 27) {
                s_rstart[2 * lane] = start;
                s_rstart[2 * lane + 1] = gs;
                s_rpre[2 * lane] = ex;
                s_rpre[2 * lane + 1] = ex + len;
            }
        } else {
            // a row's start is its first cell with atoms
            const int l1 = __shfl_down_sync(0xffffffffu, len, 1);
            const int s1 = __shfl_down_sync(0xffffffffu, start, 1), s2 = __shfl_down_sync(0xffffffffu, start, 2);
            if (lane < 27 && lane % 3 == 0) {
                s_rstart[lane / 3] = len ? start : (l1 ? s1 : s2);
                s_rpre[lane / 3] = ex;
            }
        }
        if (lane == 26) {
            s_rpre[ghosts ? 54 : 9] = incl;
            s_nr = ghosts ? 54 : 9;
        }
    }

    uint32_t* buf = s_buf[wid];
    int maxcnt = 0;

    for (int hb = h0; hb < h1; hb += 32) {
        const int hn = min(32, h1 - hb);
        if (hb > h0) __syncthreads();  // every warp has left the previous homes
        if (wid == kNlWarps - 1) {
            // the homes and their bounding box, relative to the cell's centre
            const bool home = lane < hn;
            const int i = hb + (home ? lane : 0);
            const double4 p = ldg_d4(pos + i);
            const int rb = __ldg(rbk + i), rb0 = __ldg(rbk + h0);
            const int cz = c / a.nxy, cy = (c - cz * a.nxy) / a.nx, cx = c - cz * a.nxy - cy * a.nx;
            const double ox = a.alo[0] + ((double)cx + 0.5) * a.spacing, oy = a.alo[1] + ((double)cy + 0.5) * a.spacing,
                         oz = a.alo[2] + ((double)cz + 0.5) * a.spacing;
            const float hx = (float)(p.x - ox), hy = (float)(p.y - oy), hz = (float)(p.z - oz);
            if (home) {
                s_home[lane] = make_float4(hx, hy, hz, __int_as_float(rel_code(rb, rb0)));
                if (HM) s_href[lane] = __ldg(ref + i);
                s_cnt[lane] = 0;
            }
            const float lx = warp_min(hx), ly = warp_min(hy), lz = warp_min(hz);
            const float ux = -warp_min(-hx), uy = -warp_min(-hy), uz = -warp_min(-hz);
            if (lane == 0) {
                const float mag = fmaxf(fmaxf(fmaxf(-lx, ux), fmaxf(-ly, uy)), fmaxf(-lz, uz)) + a.cut;
                const float margin = margin32(a.cut, mag), cut2 = a.cut * a.cut;
                s_box[0] = make_float4(lx, ly, lz, cut2 - margin);
                s_box[1] = make_float4(ux, uy, uz, cut2 + margin);
                s_ctr[0] = ox;
                s_ctr[1] = oy;
                s_ctr[2] = oz;
                s_rb0 = rb0;
            }
        }
        __syncthreads();  // ranges and homes are in place
        const int nr = s_nr, M = s_rpre[nr];
        if (!(s_box[1].w < a.wide2)) {
            maxcnt = max(maxcnt, far_homes<HM>(pos, ref, rbk, nbn, nbl, a.cut2, a.nbcap, a.stride, a.two ? a.N : 0, hb, hn,
                                               nr, s_rstart, s_rpre));
            continue;
        }

        for (int t0 = 0; t0 < M; t0 += kNlTile) {
            // the slots of the tile's candidates, range by range
            const int t1 = min(t0 + kNlTile, M);
            for (int r = wid; r < nr; r += kNlWarps) {
                const int first = s_rpre[r], m1 = min(s_rpre[r + 1], t1);
                const int slot = s_rstart[r] - first;
                for (int m = max(first, t0) + lane; m < m1; m += 32) s_slot[m - t0] = slot + m;
            }
            __syncthreads();
            // this warp's share of the tile, a whole number of chunks, kept in registers until the
            // warps before it know how many they keep
            const int share = ((t1 - t0 + kNlThreads - 1) / kNlThreads) * 32;
            const int m0 = wid * share, m1 = min(m0 + share, t1 - t0);
            const float4 lo = s_box[0], hi = s_box[1];
            const double ox = s_ctr[0], oy = s_ctr[1], oz = s_ctr[2];
            const int rb0 = s_rb0;  // rebasing cells are staged relative to the first home's
            float4 cp[kNlChunks];
            int cref[HM ? kNlChunks : 1];
            unsigned bal[kNlChunks];
            int kept = 0;
#pragma unroll
            for (int u = 0; u < kNlChunks; ++u) {
                bal[u] = 0u;
                if (m0 + 32 * u >= m1) continue;  // warp-uniform
                const int m = m0 + 32 * u + lane;
                const int slot = s_slot[min(m, m1 - 1)];
                const double4 p = ldg_d4(pos + slot);
                const int kb = __ldg(rbk + slot);
                // root reference index (ref for locals), below every home's where locals always pass
                if (HM) cref[u] = a.two && slot < a.N ? -1 : __ldg(ref + slot);
                cp[u] = make_float4((float)(p.x - ox), (float)(p.y - oy), (float)(p.z - oz),
                                    __uint_as_float(((uint32_t)slot << kCodeBits) +
                                                    (uint32_t)(rel_code(kb, rb0) + kCodeBias)));
                const float ex = fmaxf(fmaxf(lo.x - cp[u].x, cp[u].x - hi.x), 0.f);
                const float ey = fmaxf(fmaxf(lo.y - cp[u].y, cp[u].y - hi.y), 0.f);
                const float ez = fmaxf(fmaxf(lo.z - cp[u].z, cp[u].z - hi.z), 0.f);
                bal[u] = __ballot_sync(0xffffffffu, m < m1 && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= hi.w);
                kept += __popc(bal[u]);
            }
            if (lane == 0) s_kept[wid] = kept;
            __syncthreads();  // the shares are known, and every warp has left the previous tile
            int at = 0, nk = 0;
#pragma unroll
            for (int w = 0; w < kNlWarps; ++w) {
                const int kw = s_kept[w];
                at += w < wid ? kw : 0;
                nk += kw;
            }
#pragma unroll
            for (int u = 0; u < kNlChunks; ++u) {
                if ((bal[u] >> lane) & 1u) {
                    const int k = at + __popc(bal[u] & lt);
                    s_cand[k] = cp[u];
                    if (HM) s_cref[k] = cref[u];
                }
                at += __popc(bal[u]);
            }
            if (wid == kNlWarps - 1) {  // the last step filled up with candidates that nothing is near
#pragma unroll
                for (int u = 0; u < kNlStep; ++u) {
                    s_cand[nk + 32 * u + lane] = make_float4(1e18f, 1e18f, 1e18f, 0.f);
                    if (HM) s_cref[nk + 32 * u + lane] = 0x7fffffff;
                }
            }
            __syncthreads();

            const bool last = t1 == M;
            const float lo2 = lo.w, hi2 = hi.w;
            const uint32_t cand0 = smem_addr(&s_cand[lane]), cand_end = smem_addr(&s_cand[0]) + 16 * nk + 16 * lane;
            const uint32_t cref0 = smem_addr(&s_cref[HM ? lane : 0]);
            const uint32_t buf0 = smem_addr(buf), buf_full = buf0 + 4 * 128;
            for (int h = wid; h < hn; h += kNlWarps) {
                const float4 hp = s_home[h];
                const int i = hb + h;
                const uint32_t irel = __float_as_uint(hp.w);
                // a candidate's staged w minus irel is the entry slot << 6 | code; it equals i6 only
                // for the home itself (within the cutoff the two rebasing parts differ by less than 64)
                const uint32_t i6 = ((uint32_t)i << kCodeBits) + (uint32_t)((int)irel + kCodeBias);
                const int iref = HM ? s_href[HM ? h : 0] : 0;
                int out = M > kNlTile ? s_cnt[h] : 0;  // entries already in the list
                uint32_t bp = buf0;                       // where the next entry goes in the buffer
                uint32_t cp0 = cand0, cr0 = cref0;        // the lane's candidate of this step
                for (;;) {
                    bool take[kNlStep], near = false, may[kNlStep], slow;
                    uint32_t entry[kNlStep];
                    for (; cp0 < cand_end; cp0 += 512 * kNlStep, cr0 += 128 * kNlStep) {
                        near = bp >= buf_full;
#pragma unroll
                        for (int u = 0; u < kNlStep; ++u) {
                            const float4 q = lds_f4(cp0 + 512 * u);
                            const float dx = hp.x - q.x, dy = hp.y - q.y, dz = hp.z - q.z;
                            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                            const uint32_t s6 = __float_as_uint(q.w);
                            // the entry slot << 6 | code: the list cutoff below the rebasing spacing
                            // keeps every |dk| <= 1 within it (checked on the host)
                            entry[u] = s6 - irel;
                            // core/neighborlist.impala:34: half lists keep i > j (reference index); HM ==
                            // 2 compares ghosts by their root so pairs across the periodic boundary are
                            // kept once
                            may[u] = s6 != i6 && (!HM || lds_i(cr0 + 128 * u) < iref);
                            const bool in = r2 < lo2;
                            take[u] = may[u] && in;
                            near = near || (!in && r2 <= hi2);
                        }
                        slow = __any_sync(0xffffffffu, near);
                        if (slow) break;
#pragma unroll
                        for (int u = 0; u < kNlStep; ++u) {
                            const unsigned hits = __ballot_sync(0xffffffffu, take[u]);
                            if (take[u]) sts_u(bp + 4 * __popc(hits & lt), entry[u]);
                            bp += 4 * __popc(hits);
                        }
                    }
                    if (cp0 >= cand_end) break;
                    // a step with a pair near the cutoff, or a full buffer (kept out of the loop above,
                    // where the compiler would run all of this predicated on every step)
                    if (bp >= buf_full) {
                        int nb = (int)(bp - buf0) >> 2;
                        drain(buf, nb, out, i, nbl, a, lane);
                        bp = buf0 + 4 * nb;
                    }
#pragma unroll
                    for (int u = 0; u < kNlStep; ++u) {
                        const float4 q = lds_f4(cp0 + 512 * u);
                        const float dx = hp.x - q.x, dy = hp.y - q.y, dz = hp.z - q.z;
                        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                        bool in = r2 < lo2;
                        // |dk| <= 1 still holds near the cutoff, so the entry's slot is the candidate's
                        if (may[u] && !in && r2 <= hi2)
                            in = exact_within(pos, i, (int)(entry[u] >> kCodeBits), a.cut2);
                        const bool t = may[u] && in;
                        const unsigned hits = __ballot_sync(0xffffffffu, t);
                        if (t) sts_u(bp + 4 * __popc(hits & lt), entry[u]);
                        bp += 4 * __popc(hits);
                    }
                    cp0 += 512 * kNlStep;
                    cr0 += 128 * kNlStep;
                }
                int nb = (int)(bp - buf0) >> 2;  // entries in the buffer
                if (nb >= 128) drain(buf, nb, out, i, nbl, a, lane);
                __syncwarp();
                if ((out & 3) == 0 && last) {
                    // the last quad's padding
                    if (lane < ((-nb) & 3)) buf[nb + lane] = ((uint32_t)i << kCodeBits) | kPadCode;
                    __syncwarp();
                    store_quads(buf, (nb + 3) & ~3, out, i, nbl, a, lane);
                } else {
                    for (int e = lane; e < nb; e += 32)
                        if (out + e < a.nbcap) nbl[nl_index(out + e, i, a.stride)] = buf[e];
                    if (last && lane < ((-(out + nb)) & 3) && out + nb + lane < a.nbcap)
                        nbl[nl_index(out + nb + lane, i, a.stride)] = ((uint32_t)i << kCodeBits) | kPadCode;
                }
                __syncwarp();  // the buffer is free for the next home
                const int cnt = out + nb;
                if (last) {
                    if (lane == 0) nbn[i] = cnt;
                    maxcnt = max(maxcnt, cnt);
                } else if (lane == 0) {
                    s_cnt[h] = cnt;
                }
            }
        }
    }
    if (lane == 0 && maxcnt > 0) atomicMax(&st->max_nb, maxcnt);
}

// Sparse cells (DEM grains: ~3 to a cell and ~90 in its stencil): eight lanes to a home, four homes
// to a warp.  A home's lanes lay its stencil's ranges of slots end to end (9 rows, or 54 ranges where
// ghosts are around) and test eight candidates at once with the reference's FP64 test; the ballot
// among them places the hits.  Bound by instruction issue and
// latency (65 %, ~1,000 warp instructions per four homes).  The kernel above gives each cell a block,
// most of it idle here: contact DEM, before (a warp per cell) -> now, us: 260,800 grains 187 -> 86,
// 223,488 162 -> 79, 33,000 35 -> 21.  A thread per home took 88, 101 and 53 us; ballots among the
// eight lanes alone instead of the whole warp 106, 94 and 25 us.
constexpr int kSparseThreads = 128, kSparseLanes = 8;
constexpr int kSparseBatch = 2;  // candidates of a lane in flight (4: 95 us at 260,800 grains)

template <int HM>
__global__ void __launch_bounds__(kSparseThreads)
k_build_list_sparse(const double4* __restrict__ pos, const int* __restrict__ ref, const int* __restrict__ rbk,
                    const int* __restrict__ cstart, const int* __restrict__ slot_cell, int* __restrict__ nbn,
                    uint32_t* __restrict__ nbl, DevStatus* st, NlArgs a, int local_blocks, LinkArgs la) {
    const int blk = (int)blockIdx.x + pdl_wait();
    // a home's ranges: candidates before it, first slot minus that
    __shared__ int2 s_range[kSparseThreads / kSparseLanes][55];
    if (blk >= local_blocks) {  // blocks past the locals link the ghosts (k_ghost_links' work)
        const int h = (blk - local_blocks) * blockDim.x + threadIdx.x;
        if (h < la.G) ghost_link(h, la);
        return;
    }
    const int lane = threadIdx.x & 31, l = lane % kSparseLanes;
    const int i = (blk * kSparseThreads + threadIdx.x) / kSparseLanes;
    const unsigned group = 0xffu << (lane - l), before = lanemask_lt() & group;
    int cnt = 0;
    // a home outside the grid (or past the last one) has no candidates; the warp's homes keep together,
    // so that shuffles and ballots run over whole warps
    const int c = i < a.N ? slot_cell[i] : a.ncells;
    const bool act = c < a.ncells;
    const int ih = act ? i : 0;
    const double4 pi = ldg_d4(pos + ih);
    const int rb = __ldg(rbk + ih);
    const int iref = HM ? __ldg(ref + ih) : 0;
    const int* gstart = cstart + a.ncells + 1;
    int2* range = s_range[threadIdx.x / kSparseLanes];
    // lane l takes row l of the stencil, all lanes row 8
    int len[2], start[2];
    bool ghosts = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int r = q ? 8 : l;
        const int row = c + (r / 3 - 1) * a.nxy + (r % 3 - 1) * a.nx;
        const int c0 = min(max(row - 1, 0), a.ncells), c1 = act ? min(max(row + 2, 0), a.ncells) : c0;
        start[q] = __ldg(cstart + c0);
        len[q] = __ldg(cstart + c1) - start[q];
        ghosts = ghosts || __ldg(gstart + c0) != __ldg(gstart + c1);
    }
    int M;
    if (!__any_sync(0xffffffffu, ghosts)) {
        int incl = len[0];
#pragma unroll
        for (int o = 1; o < kSparseLanes; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o, kSparseLanes);
            if (l >= o) incl += y;
        }
        range[l] = make_int2(incl - len[0], start[0] - (incl - len[0]));
        if (l == kSparseLanes - 1) range[8] = make_int2(incl, start[1] - incl);
        M = __shfl_sync(0xffffffffu, incl, kSparseLanes - 1, kSparseLanes) + len[1];
        if (l == 0) range[9] = make_int2(M, 0);
    } else {  // cell by cell, the locals then the ghosts of each
        M = 0;
        for (int k0 = 0; k0 < 27; k0 += kSparseLanes) {
            const int k = k0 + l, nb = c + (k / 9 - 1) * a.nxy + ((k / 3) % 3 - 1) * a.nx + k % 3 - 1;
            int ls = 0, ll = 0, gs = 0, gl = 0;
            if (act && k < 27 && nb >= 0 && nb < a.ncells) {
                ls = __ldg(cstart + nb);
                ll = __ldg(cstart + nb + 1) - ls;
                gs = __ldg(gstart + nb);
                gl = __ldg(gstart + nb + 1) - gs;
            }
            int incl = ll + gl;
#pragma unroll
            for (int o = 1; o < kSparseLanes; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o, kSparseLanes);
                if (l >= o) incl += y;
            }
            const int ex = M + incl - ll - gl;
            if (k < 27) {
                range[2 * k] = make_int2(ex, ls - ex);
                range[2 * k + 1] = make_int2(ex + ll, gs - ex - ll);
            }
            M += __shfl_sync(0xffffffffu, incl, kSparseLanes - 1, kSparseLanes);
        }
        if (l == 0) range[54] = make_int2(M, 0);
    }
    __syncwarp();
    const int most = __reduce_max_sync(0xffffffffu, M);
    int r = 0, rend = range[1].x, roff = range[0].y;
    for (int m0 = l; m0 - l < most; m0 += kSparseLanes * kSparseBatch) {
        // positions, rebasing cells and keys of a batch load together
        double4 p[kSparseBatch];
        int slot[kSparseBatch], kb[kSparseBatch], kr[HM ? kSparseBatch : 1];
#pragma unroll
        for (int u = 0; u < kSparseBatch; ++u) {
            const int m = m0 + u * kSparseLanes;
            if (m < M) {
                while (rend <= m) {
                    ++r;
                    rend = range[r + 1].x;
                    roff = range[r].y;
                }
            }
            slot[u] = m < M ? m + roff : ih;
            p[u] = ldg_d4(pos + slot[u]);
            kb[u] = __ldg(rbk + slot[u]);
            if (HM) kr[u] = a.two && slot[u] < a.N ? -1 : __ldg(ref + slot[u]);
        }
#pragma unroll
        for (int u = 0; u < kSparseBatch; ++u) {
            const double r2 = len2_strict(dsub(pi.x, p[u].x), dsub(pi.y, p[u].y), dsub(pi.z, p[u].z));
            // core/neighborlist.impala:34: half lists keep i > j (reference index); HM == 2 compares
            // ghosts by their root
            const bool take = r2 <= a.cut2 && slot[u] != ih && (!HM || kr[HM ? u : 0] < iref);
            const unsigned hits = __ballot_sync(0xffffffffu, take) & group;
            const int k = cnt + __popc(hits & before);
            if (take && k < a.nbcap)
                nbl[nl_index(k, i, a.stride)] =
                    ((uint32_t)slot[u] << kCodeBits) + (uint32_t)(rel_code(kb[u], rb) + kCodeBias);
            cnt += __popc(hits);
        }
    }
    // the last quad's padding
    if (act && l < ((-cnt) & 3) && cnt + l < a.nbcap)
        nbl[nl_index(cnt + l, i, a.stride)] = ((uint32_t)i << kCodeBits) | kPadCode;
    if (i < a.N && l == 0) nbn[i] = cnt;
    cnt = warp_max(cnt);
    if (lane == 0 && cnt > 0) atomicMax(&st->max_nb, cnt);
}

// Locals outside the grid (bucket ncells) get empty lists.
__global__ void k_clear_lists(int* __restrict__ nbn, int a, int b) {
    const int blk = (int)blockIdx.x + pdl_wait();
    int i = a + blk * blockDim.x + threadIdx.x;
    if (i < b) nbn[i] = 0;
}

// ---- exclusive scan ------------------------------------------------------------
__device__ __forceinline__ int block_exscan(int v, int* total, int* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int nw = blockDim.x >> 5;
        int w = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sh[lane] = w;  // inclusive prefix of warp sums
    }
    __syncthreads();
    int r = x - v + (wid ? sh[wid - 1] : 0);
    *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return r;
}

constexpr int kScanThreads = 1024, kScanItems = 4, kScanBlock = kScanThreads * kScanItems;

// per-block totals of the input
__global__ void k_scan_sums(const int* __restrict__ in, int* __restrict__ part, int n) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ int sh[32];
    int base = blk * kScanBlock + threadIdx.x * kScanItems;
    int s = 0;
    for (int k = 0; k < kScanItems; ++k) s += (base + k < n) ? in[base + k] : 0;
    int tot;
    block_exscan(s, &tot, sh);
    if (threadIdx.x == 0) part[blk] = tot;
}

// exclusive scan of the block totals in place (one block); part[nb] = grand total
__global__ void k_scan_part(int* __restrict__ part, int nb) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ int sh[32];
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += kScanThreads) {
        int i = b0 + threadIdx.x + blk;
        int v = i < nb ? part[i] : 0;
        int tot;
        int ex = block_exscan(v, &tot, sh);
        if (i < nb) part[i] = carry + ex;
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) part[nb] = carry;
}

__global__ void k_scan_apply(const int* __restrict__ in, int* __restrict__ out, const int* __restrict__ part,
                             int n, int nb) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ int sh[32];
    int base = blk * kScanBlock + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        s += v[k];
    }
    int tot;
    int ex = block_exscan(s, &tot, sh) + part[blk];
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = ex;
        ex += v[k];
    }
    if (blk == nb - 1 && threadIdx.x == 0) out[n] = part[nb];
}

// Exclusive scan of up to kScanSingleMax values in one block: the values are staged in
// shared memory by coalesced loads, each thread scans a run of consecutive values there,
// the block scans the run totals, and the results leave by coalesced stores.  One launch
// instead of three for the counts of a rebuild (tens of thousands of values).
constexpr int kScanSingleMax = 32768;  // 128 KiB of shared memory
__global__ void __launch_bounds__(kScanThreads) k_scan_single(const int* __restrict__ in, int* __restrict__ out,
                                                               int n) {
    const int blk = (int)blockIdx.x + pdl_wait();
    extern __shared__ int sv[];
    __shared__ int sh[32];
#pragma unroll 8
    for (int k = threadIdx.x + blk; k < n; k += kScanThreads) sv[k] = in[k];
    __syncthreads();
    const int run = (n + kScanThreads - 1) / kScanThreads;
    const int base = threadIdx.x * run;
    const int end = min(base + run, n);
    int s = 0;
    for (int k = base; k < end; ++k) s += sv[k];
    int tot;
    int ex = block_exscan(s, &tot, sh);
    for (int k = base; k < end; ++k) {
        const int v = sv[k];
        sv[k] = ex;
        ex += v;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = threadIdx.x; k < n; k += kScanThreads) out[k] = sv[k];
    if (threadIdx.x == 0) out[n] = tot;
}

// ---- host wrappers ---------------------------------------------------------------
// Single-pass exclusive scan of a long array (decoupled look-back): block b scans tile b,
// publishes its total, then adds the totals of the tiles before it -- a tile that already
// knows its inclusive prefix ends the walk -- and publishes that prefix.  A tile word holds
// (launch epoch << 2 | state) << 32 | value, so nothing is reset between launches.  The wait
// for a predecessor is bounded: past the limit the block sums that predecessor's inputs (and
// all before it) directly, so the result never depends on the wait ending (the grids here
// are a few dozen blocks, all resident at once).  One launch with ~11 blocks for the 21k cell
// counts of a 131k-atom rebuild, where one block walked all of them.
constexpr int kLbThreads = 256, kLbItems = 8, kLbTile = kLbThreads * kLbItems;
constexpr int kLbSpinLimit = 1 << 14;  // polls of a predecessor's word (64 ns apart) before summing it directly

__device__ __forceinline__ unsigned long long lb_word(unsigned epoch, unsigned state, int v) {
    return ((unsigned long long)((epoch << 2) | state) << 32) | (unsigned)v;
}

__global__ void __launch_bounds__(kLbThreads)
k_scan_lookback(const int* __restrict__ in, int* __restrict__ out, int n, int ntiles,
                unsigned long long* __restrict__ tiles, unsigned epoch) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ int sh[32];
    __shared__ int s_prefix, s_missing;
    const int tile = blk;
    const int base = tile * kLbTile + threadIdx.x * kLbItems;
    int v[kLbItems];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < kLbItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        sum += v[k];
    }
    int total;
    const int ex = block_exscan(sum, &total, sh);
    if (threadIdx.x == 0) {
        int excl = 0, missing = -1;
        volatile unsigned long long* tw = tiles;
        if (tile == 0) {
            tw[0] = lb_word(epoch, 2u, total);
        } else {
            tw[tile] = lb_word(epoch, 1u, total);
            const unsigned want = epoch & 0x3fffffffu;
            for (int j = tile - 1; j >= 0; --j) {
                unsigned long long w = tw[j];
                int spins = 0;
                while (((unsigned)(w >> 34) != want || ((w >> 32) & 3u) == 0u) && spins < kLbSpinLimit) {
                    __nanosleep(64);
                    w = tw[j];
                    ++spins;
                }
                if ((unsigned)(w >> 34) != want || ((w >> 32) & 3u) == 0u) {
                    missing = j;
                    break;
                }
                excl += (int)(unsigned)w;
                if (((w >> 32) & 3u) == 2u) break;
            }
            if (missing < 0) tw[tile] = lb_word(epoch, 2u, excl + total);
        }
        s_prefix = excl;
        s_missing = missing;
    }
    __syncthreads();
    int prefix = s_prefix;
    if (s_missing >= 0) {  // the inputs of tiles 0..missing summed directly
        const int end = min(n, (s_missing + 1) * kLbTile);
        int part = 0;
        for (int i = threadIdx.x; i < end; i += kLbThreads) part += in[i];
        int all;
        block_exscan(part, &all, sh);
        prefix += all;
        if (threadIdx.x == 0) ((volatile unsigned long long*)tiles)[tile] = lb_word(epoch, 2u, prefix + total);
    }
    int e = prefix + ex;
#pragma unroll
    for (int k = 0; k < kLbItems; ++k) {
        if (base + k < n) out[base + k] = e;
        e += v[k];
    }
    if (tile == ntiles - 1 && threadIdx.x == 0) out[n] = prefix + total;
}

static inline int nblocks(long long n, int t) { return (int)((n + t - 1) / t); }

void ensure_scan_scratch(State& s, int n) {
    int nb = nblocks(n, kScanBlock) + 1;
    if (nb > s.scan_part_cap) {
        dfree(&s.scan_part);
        s.scan_part_cap = nb + 64;
        dalloc(&s.scan_part, s.scan_part_cap);
    }
}

// look-back scans from this many values on (below, one block is as fast)
#ifndef TMD_LB_MIN
#define TMD_LB_MIN 8192
#endif
constexpr int kLookbackMin = TMD_LB_MIN;

static bool ensure_lookback(State& s, int ntiles) {
    if (ntiles <= s.lb_tile_cap) return true;
    dfree(&s.lb_tiles);
    s.lb_tile_cap = ntiles + 64;
    dalloc(&s.lb_tiles, s.lb_tile_cap);
    if (!s.lb_tiles) {
        s.lb_tile_cap = 0;
        return false;
    }
    TMD_CUDA(cudaMemsetAsync(s.lb_tiles, 0, sizeof(unsigned long long) * s.lb_tile_cap, s.stream));
    return true;
}

// out[0..n-1] = exclusive prefix sums of in, out[n] = total (in != out allowed only)
void exclusive_scan(State& s, const int* in, int* out, int n) {
    if (n >= kLookbackMin) {
        const int ntiles = nblocks(n, kLbTile);
        if (ensure_lookback(s, ntiles)) {
            launch(s, ntiles, kLbThreads, 0, k_scan_lookback, in, out, n, ntiles, s.lb_tiles, ++s.lb_epoch);
            launched(K_SCAN);
            return;
        }
    }
    if (n <= kScanSingleMax) {
        if (s.scan_attr_device != s.device) {  // a function attribute is set per device
            TMD_CUDA(cudaFuncSetAttribute(k_scan_single, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kScanSingleMax * (int)sizeof(int)));
            s.scan_attr_device = s.device;
        }
        launch(s, 1, kScanThreads, (size_t)n * sizeof(int), k_scan_single, in, out, n);
        launched(K_SCAN);
        return;
    }
    int nb = nblocks(n, kScanBlock);
    if (nb < 1) nb = 1;
    ensure_scan_scratch(s, n);
    launch(s, nb, kScanThreads, 0, k_scan_sums, in, s.scan_part, n);
    launched(K_SCAN);
    launch(s, 1, kScanThreads, 0, k_scan_part, s.scan_part, nb);
    launched(K_SCAN);
    launch(s, nb, kScanThreads, 0, k_scan_apply, in, out, s.scan_part, n, nb);
    launched(K_SCAN);
}

void run_enforce_pbc(State& s) {
    if (s.N == 0) return;
    GeoArgs a = geo_args(s.geo);
    prof_begin(K_PBC);
    launch(s, nblocks(s.N, 256), 256, 0, k_enforce_pbc, s.pos.b[s.pc], s.img.b[s.ac], s.N, a);
    launched(K_PBC);
    prof_end(K_PBC);
}

bool grow_atoms(State& s, int need);  // api.cu

// Words of HostStatus that a kernel in flight stores, polled for: the host goes on a few microseconds
// earlier than after a copy and an event, and the kernels keep following one another without either
// between them.  When they do not come (a failed launch, a long queue ahead) the stream's work is
// waited for.  A rebuild of eight kernels with two such waits, by copies and events -> by words stored (us
// on top of an ordinary step): 256 atoms 54 -> 40, 2,048 55 -> 40, 16,384 65 -> 51, 131,072 143 -> 130,
// half-filled box of 524,288 433 -> 421, granular gas of 260,800 162 -> 147; at a rebuild every 20 steps
// 7.24 -> 6.44 us a step at 256 atoms, 14.0 -> 13.4 at 16,384, 44.4 -> 43.5 at 131,072.  A fence after
// the stores, with one word for all of them, took 2 us.
bool await_words(State& s, void* words, int n) {
    const volatile int* const w = static_cast<const volatile int*>(words);
    const auto start = std::chrono::steady_clock::now();
    int k = 0;
    for (unsigned polls = 1; k < n; ++polls) {
        while (k < n && w[k] >= 0) ++k;
        if ((polls & 0xfffu) == 0 && std::chrono::steady_clock::now() - start > std::chrono::seconds(1)) break;
    }
    if (k < n) TMD_CUDA(cudaStreamSynchronize(s.stream));
    std::atomic_thread_fence(std::memory_order_acquire);
    while (k < n && w[k] >= 0) ++k;
    return k == n;
}

void run_borders(State& s, bool wrap) {
    GeoArgs a = geo_args(s.geo);
    const int N = s.N;
    const int nblk = border_blocks(N);
    if (N == 0 && !s.halo.on) {
        s.G = 0;
        return;
    }
    prof_begin(K_BORDER);
    const int nseg = 2 * (a.ncells + 1);
    const int n = 26 * nblk;
    // boff = exclusive scan of bcount, stored after the counts
    int* boff = s.bcount + n;
    if (s.halo.on) {
        // several ranks: the per-type totals first (they split the images into this rank's
        // periodic ghosts and the ones for other ranks), then the emit, then the exchange;
        // a rank without locals still takes part in the exchange
        if (N > 0) {
            if (wrap)
                launch(s, nblk, kBorderThreads, 0, k_border_count<true>, s.pos.b[s.pc], s.img.b[s.ac], s.slot_of_ref,
                       s.bmask, s.bcount, N, nblk, a, s.cnt, nseg, s.status_dev);
            else
                launch(s, nblk, kBorderThreads, 0, k_border_count<false>, s.pos.b[s.pc], s.img.b[s.ac],
                       s.slot_of_ref, s.bmask, s.bcount, N, nblk, a, s.cnt, nseg, s.status_dev);
            s.bin_zeroed = true;
            launched(K_BORDER);
            exclusive_scan(s, s.bcount, boff, n);
        }
        bool ok = halo_plan_borders(s, N > 0 ? boff : nullptr, nblk);
        if (ok && N + s.halo.gself > s.capA) ok = grow_atoms(s, N + s.halo.gself);
        if (ok && N > 0) {
            RemoteOut ro{s.halo.tab, s.halo.send_ref, s.halo.send_type, comm().topo.selfmask};
            launch(s, nblk, kBorderThreads, 0, k_border_emit<true>, s.pos.b[s.pc], s.vel.b[s.vc], s.frc.b[s.ac],
                   s.mass.b[s.ac], s.ref.b[s.ac], s.slot_of_ref, s.bmask, boff, s.gsrc, s.groot, s.gcode, s.bsrc_ref,
                   s.broot_ref, s.bcode, N, nblk, s.capA, a, s.dem_fixed, ro, nullptr);
            launched(K_BORDER);
        }
        if (ok) ok = halo_finish_borders(s);
        if (!ok) s.G = 0;
        prof_end(K_BORDER);
        s.lists_valid = 0;
        return;
    }
    if (wrap)
        launch(s, nblk, kBorderThreads, 0, k_border_count<true>, s.pos.b[s.pc], s.img.b[s.ac], s.slot_of_ref,
               s.bmask, s.bcount, N, nblk, a, s.cnt, nseg, s.status_dev);
    else
        launch(s, nblk, kBorderThreads, 0, k_border_count<false>, s.pos.b[s.pc], s.img.b[s.ac], s.slot_of_ref,
               s.bmask, s.bcount, N, nblk, a, s.cnt, nseg, s.status_dev);
    s.bin_zeroed = true;
    launched(K_BORDER);
    exclusive_scan(s, s.bcount, boff, n);
    // The ghost count comes back while the emit kernel already runs: emit writes only the
    // slots below the capacity, so when the count shows the capacity was short the host
    // grows the arrays (which waits for that emit) and emits again.  The host thus enqueues
    // the next kernels before emit finishes instead of leaving the GPU idle for a round trip.
    // Emit's first thread stores the count straight to page-locked memory (await_words).
    auto emit = [&](int* count) {
        launch(s, nblk, kBorderThreads, 0, k_border_emit<false>, s.pos.b[s.pc], s.vel.b[s.vc], s.frc.b[s.ac],
               s.mass.b[s.ac], s.ref.b[s.ac], s.slot_of_ref, s.bmask, boff, s.gsrc, s.groot, s.gcode, s.bsrc_ref,
               s.broot_ref, s.bcode, N, nblk, s.capA, a, s.dem_fixed, RemoteOut{nullptr, nullptr, nullptr, 0u}, count);
        launched(K_BORDER);
    };
    int* const count = &s.status_host->nghost;
    *static_cast<volatile int*>(count) = -1;
    emit(count);
    if (!await_words(s, count, 1)) {  // a latched error
        s.G = 0;
        s.lists_valid = 0;
        prof_end(K_BORDER);
        return;
    }
    const int G = *static_cast<volatile int*>(count);
    if (N + G > s.capA) {
        if (!grow_atoms(s, N + G)) {  // no room: no ghosts rather than writes past the arrays
            s.G = 0;
            s.lists_valid = 0;
            prof_end(K_BORDER);
            return;
        }
        emit(nullptr);
    }
    prof_end(K_BORDER);
    s.G = G;
    s.lists_valid = 0;
}

void run_distribute(State& s) {
    GeoArgs a = geo_args(s.geo);
    const int N = s.N, NA = s.N + s.G;
    const int nseg = 2 * (a.ncells + 1);
    if (NA == 0) return;
    prof_begin(K_BIN);
    if (!s.bin_zeroed) {  // else zeroed by the border pass's first kernel
        TMD_CUDA(cudaMemsetAsync(s.cnt, 0, sizeof(int) * nseg, s.stream));
        TMD_CUDA(cudaMemsetAsync(&s.status_dev->out_local, 0, 6 * sizeof(int), s.stream));  // .. filled
    }
    s.bin_zeroed = false;
    launch(s, nblocks(NA, 256), 256, 0, k_bin_count, s.pos.b[s.pc], s.cnt, s.bin_cell, s.bin_rank, s.status_dev, N,
           NA, a);
    launched(K_BIN);
    exclusive_scan(s, s.cnt, s.cstart, nseg);
    launch(s, nblocks(NA, 256), 256, 0, k_bin_scatter, s.ref.b[s.ac], s.bin_cell, s.bin_rank, s.cstart, s.tmp_key,
           s.tmp_src, N, NA, a.ncells);
    launched(K_BIN);
    const int np = 1 - s.pc, nv = 1 - s.vc, na = 1 - s.ac;
    MoveArgs m;
    m.pos_o = s.pos.b[s.pc]; m.pos_n = s.pos.b[np];
    m.vel_o = s.vel.b[s.vc]; m.vel_n = s.vel.b[nv];
    m.frc_o = s.frc.b[s.ac]; m.frc_n = s.frc.b[na];
    m.mass_o = s.mass.b[s.ac]; m.mass_n = s.mass.b[na];
    m.ref_o = s.ref.b[s.ac]; m.ref_n = s.ref.b[na];
    m.img_o = s.img.b[s.ac]; m.img_n = s.img.b[na];
    m.slot_of_ref = s.slot_of_ref; m.rref = s.rref; m.rbk = s.rbk;
    m.bin_cell = s.bin_cell; m.slot_cell = s.slot_cell;
    m.pos32 = s.pos32.b[np]; m.img_cnt = s.img_cnt; m.img_slot = s.img_slot;
    m.capA = s.capA; m.N = N; m.mixed = s.precision;
    launch(s, nblocks(NA, 256), 256, 0, k_rank_move, s.cstart, s.tmp_key, s.tmp_src, NA, a.ncells, m, a,
           s.status_dev);
    launched(K_BIN);
    s.build_zeroed = true;
    s.pc = np;
    s.vc = nv;
    s.ac = na;
    // the ghost links run as extra blocks of the list build that follows, or alone
    // (flush_links) before anything else that reads them
    s.pend_links = s.G > 0;
    s.img_ok = 0;  // known after the status readback of the list build
    s.nchain = 0;
    prof_end(K_BIN);
    s.lists_valid = 0;
}

void grow_lists(State& s, int rows);  // api.cu

LinkArgs link_args(State& s) {
    LinkArgs l;
    l.ref = s.ref.b[s.ac];
    l.slot_of_ref = s.slot_of_ref;
    l.bsrc_ref = s.bsrc_ref;
    l.broot_ref = s.broot_ref;
    l.bcode = s.bcode;
    l.gsrc = s.gsrc;
    l.groot = s.groot;
    l.gcode = s.gcode;
    l.rref = s.rref;
    l.img_cnt = s.img_cnt;
    l.img_slot = s.img_slot;
    l.chain = s.chain;
    l.st = s.status_dev;
    l.N = s.N;
    l.G = s.G;
    l.capA = s.capA;
    return l;
}

void flush_links(State& s) {
    if (!s.pend_links) return;
    s.pend_links = false;
    launch(s, nblocks(s.G, 256), 256, 0, k_ghost_links, link_args(s));
    launched(K_BIN);
}

// Which list kernel: a block per cell from 8.5 locals per filled cell on.  Measured on LJ liquids of
// 131,072 atoms with smaller cutoffs, block per cell / eight lanes per home, us: 2.8 per cell 158 / 53,
// 4.9 112 / 69, 7.8 94 / 87, 11.7 85 / 112, 18.5 91 / 158; the same line at 16,384 and 442,368 atoms.
// Below 4,096 locals the block per cell is as fast or faster at every density where few cells are empty.
// An empty cell's block costs 0.52 ns, one that holds few locals 2 ns, so the eight lanes take over where
// that outweighs their longer chain (up to 9 us, by density) and their cost per home at high density.
// Gas of 500 locals in 148,877 cells 82 / 8.6 us, of 4,000 in 6,859 21 / 10.7; a liquid cluster of 4,000 in
// 32,768 25.0 / 21.2, in 148,877 82 / 21, of 32,000 in 32,768 37 / 44, in 59,319 48 / 43, of 108,000 in
// 97,336 101 / 111, in 148,877 125 / 111.  (A warp per cell, as earlier: 25, 12.7, 49, 57, 59, 62, 110, 111.)
// The filled cells are those of the last binning whose status was read (the results are the same either
// way); before the first one the box's mean density stands in, at most a cell per local.
static bool sparse_cells(const State& s) {
    const Geometry& g = s.geo;
    const double box = g.len[0] * g.len[1] * g.len[2] / (g.spacing * g.spacing * g.spacing);
    const double filled = s.cells_filled > 0 ? s.cells_filled : std::min((double)s.N, box);
    const double each = s.N / filled, over = each - 8.5;
    if (s.N > 4096 && over < 0.0) return true;
    const double saved = 0.52 * (g.ncells - filled) + (over < 0.0 ? 1.5 * filled : 0.0);  // ns
    return saved > 2000.0 + 500.0 * each + 0.05 * s.N * std::max(over, 0.0);
}

template <int HM>
void launch_build_list(State& s, const int* ref, const NlArgs& a, const LinkArgs& la, int links) {
    const int lb = nblocks(links, kNlThreads);
    if (sparse_cells(s)) {
        const int nb = nblocks((long long)s.N * kSparseLanes, kSparseThreads);
        launch(s, nb + lb, kSparseThreads, 0, k_build_list_sparse<HM>, s.pos.b[s.pc], ref, s.rbk, s.cstart,
               s.slot_cell, s.nbn, s.nbl, s.status_dev, a, nb, la);
    } else {
        launch(s, a.ncells + lb, kNlThreads, 0, k_build_list<HM>, s.pos.b[s.pc], ref, s.rbk, s.cstart, s.nbn, s.nbl,
               s.status_dev, a, a.ncells, la);
    }
}

// Half lists whose local pairs are held by both atoms (a ghost pair still by one), for the FP64 LJ
// kernel: it then adds up each atom's own pairs and only a ghost's root gets its reaction by atomics,
// where three FP64 atomics per pair, 15 M a step at 131,072 atoms, took half of the step; and few atoms
// can share each atom's list between lanes.  Step times in us, one-sided -> two-sided (boundary pairs
// kept, rebuild every 20 steps included): 256 atoms 26.8 -> 10.8, 2,048 27.3 -> 11.7, 16,384 28.2 -> 18.9,
// 48,668 44.3 -> 37.9, 131,072 83.1 -> 57.4, 442,368 240 -> 158, 864,000 447 -> 274.  The list build
// stays within 2 %.  Not for the other half kernels (DEM's lists are short, the mixed form adds four
// floats at once), nor where the longer lists outgrow the capacity of the reference's.  The force is this
// grid's last one; the lists built before its first are DEM's when the contact model is set.
static bool two_sided(const State& s) {
    const bool dem = s.force_seen ? s.force_cfg.dem : s.dem_fixed != 0;
    return s.precision == 0 && !dem && !s.two_short;
}

// Drops the entries that the reference's half lists do not hold, in place and in order: a local
// neighbour stays with the atom of the larger reference index (core/neighborlist.impala:34).
__global__ void k_one_sided(const int* __restrict__ ref, int* __restrict__ nbn, uint32_t* __restrict__ nbl, int N,
                            int stride, int nbcap) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int n = min(nbn[i], nbcap), iref = ref[i];
    int out = 0;
    for (int k = 0; k < n; ++k) {
        const uint32_t e = nbl[nl_index(k, i, stride)];
        const int j = (int)(e >> kCodeBits);
        if (j >= N || ref[j] < iref) nbl[nl_index(out++, i, stride)] = e;
    }
    nbn[i] = out;
    for (; out & 3; ++out) nbl[nl_index(out, i, stride)] = ((uint32_t)i << kCodeBits) | kPadCode;
}

void one_sided_lists(State& s) {
    if (!s.lists_two) return;
    resolve_lists(s);
    if (!s.lists_two) return;  // they outgrew the capacity and were built again
    s.lists_two = false;
    launch(s, nblocks(s.N, 256), 256, 0, k_one_sided, s.ref.b[s.ac], s.nbn, s.nbl, s.N, s.nb_stride, s.nb_cap);
    launched(K_NLIST);
}

// the list build's status to the host
__global__ void k_status_out(const DevStatus* st, HostStatus* out) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int t = threadIdx.x + blk;
    if (t < kStatusWords) reinterpret_cast<volatile int*>(&out->build)[t] = reinterpret_cast<const volatile int*>(st)[t];
}

// A list build's status, read back: the locals outside the grid get empty lists, the two-phase
// chain and image-map state of the links; 0 when the lists stand, 1 when the capacity was short
// (grown: the build is to be redone).
static int finish_build(State& s) {
    const Geometry& g = s.geo;
    if (s.status_host->build.out_local > 0) {
        int first_out = 0;
        // locals outside the grid sit at [cstart[ncells], N): empty lists
        TMD_CUDA(cudaMemcpyAsync(&first_out, s.cstart + g.ncells, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
        TMD_CUDA(cudaStreamSynchronize(s.stream));
        launch(s, nblocks(s.N - first_out, 256), 256, 0, k_clear_lists, s.nbn, first_out, s.N);
        launched(K_NLIST);
        set_error(5, "locals outside the cell grid at binning (they have no neighbours)");
    }
    s.nchain = s.status_host->build.nchain;
    s.cells_filled = s.status_host->build.filled;
    s.img_ok = (s.status_host->build.img_over1 == 0 ? 1 : 0) | (s.status_host->build.img_over2 == 0 ? 2 : 0);
    const int mx = s.status_host->build.max_nb;
    s.max_list = mx;
    if (mx <= s.nb_cap) {
        s.lists_valid = 1;
        return 0;
    }
    if (s.lists_two) {  // one-sided lists may still fit
        s.two_short = true;
        return 1;
    }
    // core/neighborlist.impala:74-76: grow to twice the overflow and redo
    std::printf("0> reallocate_neighborlist_capacity(): %d\n", mx * 2);
    grow_lists(s, mx * 2);
    return 1;
}

int run_build_lists(State& s, bool half, double cutoff, bool defer) {
    const Geometry& g = s.geo;
    s.lists_cutoff = cutoff;
    s.status_pending = false;
    if (s.N == 0) {
        s.lists_two = false;
        s.lists_valid = 1;
        s.lists_half = half;
        return 0;
    }
    // the half lists that keep boundary pairs read the ghosts' root references, which the
    // links write: they run first, alone
    if (half && s.half_ghost) flush_links(s);
    NlArgs a;
    a.cut2 = cutoff * cutoff;
    a.cut = (float)cutoff;
    a.wide2 = (float)std::max(g.rb_h * g.rb_h * (1.0 - 1e-6), a.cut2 * (1.0 + 1e-4));
    a.N = s.N;
    a.ncells = g.ncells;
    a.nx = g.nx;
    a.nxy = g.nx * g.ny;
    a.stride = s.nb_stride;
    for (int d = 0; d < 3; ++d) a.alo[d] = g.aabb_lo[d];
    a.spacing = g.spacing;
    for (int attempt = 0; attempt < 8; ++attempt) {
        a.nbcap = s.nb_cap;
        a.two = s.lists_two = half && two_sided(s);
        s.lists_half = half;  // known from the launch on: a deferred build's lists are used before its status is read
        if (attempt > 0 || !s.build_zeroed)  // else zeroed by the binning's reorder kernel
            TMD_CUDA(cudaMemsetAsync(&s.status_dev->max_nb, 0, sizeof(int), s.stream));
        s.build_zeroed = false;
        prof_begin(K_NLIST);
        // the pending ghost links ride along as extra blocks (once: they count with atomics)
        const LinkArgs la = link_args(s);
        const int links = s.pend_links ? s.G : 0;
        s.pend_links = false;
        if (half && s.half_ghost) launch_build_list<2>(s, s.rref, a, la, links);
        else if (half) launch_build_list<1>(s, s.ref.b[s.ac], a, la, links);
        else launch_build_list<0>(s, s.ref.b[s.ac], a, la, links);
        launched(K_NLIST);
        prof_end(K_NLIST);
        for (int k = 0; k < kStatusWords; ++k) reinterpret_cast<volatile int*>(&s.status_host->build)[k] = -1;
        launch(s, 1, 32, 0, k_status_out, s.status_dev, s.status_host);
        launched(K_MISC);
        if (defer && attempt == 0) {
            // the host goes on; the next force kernel is launched on these lists at once and
            // resolve_lists reads the status while it runs
            s.status_pending = true;
            s.status_half = half;
            s.lists_valid = 0;
            return 0;
        }
        TMD_CUDA(cudaStreamSynchronize(s.stream));
        if (finish_build(s) == 0) return 0;
    }
    set_error(2, "neighbour list capacity did not converge");
    return -1;
}

int resolve_lists(State& s) {
    if (!s.status_pending) return 0;
    s.status_pending = false;
    if (!await_words(s, &s.status_host->build, kStatusWords)) return -1;  // a latched error
    const bool outside = s.status_host->build.out_local > 0;
    if (finish_build(s) == 0) return outside ? 1 : 0;
    // the capacity was short: the build again, on the grown lists
    return run_build_lists(s, s.status_half, s.lists_cutoff) == 0 ? 1 : -1;
}

}  // namespace tmd
