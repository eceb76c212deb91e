// api.cu -- the md_* C ABI of the tinyMD B200 library (host orchestration).
//
// Replaces the runtime of core/runtime.impala for one process on one GPU.
// The reference synchronises after every kernel (backend/mapping_gpu.impala:
// 12-27); here calls enqueue on one stream and adjacent calls of a timestep
// are fused:
//   md_initial_integration + md_synchronize_ghost_layer -> one kernel
//   md_compute_lennard_jones (full list) + md_final_integration -> one kernel
// Every call that exposes data to the host drains pending work first.

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <deque>
#include <mutex>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "comm.h"
#include "md_common.cuh"
#include "launch.cuh"
#include "md_state.h"
#include "tinymd_b200.h"

namespace tmd {

State g_state;

// An NVTX range over an entry point that enqueues work, so a profiler's timeline (nsys, or
// `ncu --nvtx`) groups the kernels by the md_* call that issued them.  NVTX is header-only here:
// without an attached tool a range costs a pointer test.
struct Range {
    explicit Range(const char* name) { nvtxRangePushA(name); }
    ~Range() { nvtxRangePop(); }
};

// ---------------------------------------------------------------------------
// errors, launches, memory
// ---------------------------------------------------------------------------
void set_error(int code, const std::string& msg) {
    g_state.last_error = code;
    g_state.last_error_msg = msg;
    std::fprintf(stderr, "tinymd_b200: %s\n", msg.c_str());
}

bool cuda_ok(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return true;
    set_error(MD_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    return false;
}

void launched(int kernel_id) {
    (void)kernel_id;
    g_state.launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) set_error(MD_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
}

// Device blocks a closed grid leaves are kept for the next one.  A grid takes some twenty of them,
// and cudaMalloc / cudaFree cost more than a short run's steps: opening and closing a grid took 2.4
// ms at 2,048 atoms and 3.5 ms at 131,072 on a quiet host (100 steps of the mixed form: 2.1 and 3.9
// ms), and 20-50 ms where other processes of the host allocate at the same time.  Kept blocks are
// bounded in number and bytes and go back to the device at md_mpi_finalize, or at once when an
// allocation fails.  A block is handed out again only after a device synchronisation that follows
// its release, as cudaFree waits for the work that uses a block.
namespace {
struct Block {
    void* p;
    size_t bytes;
    int device;
    bool idle;  // a device synchronisation followed its release
};
constexpr size_t kKeepBytes = (size_t)1 << 30;
constexpr size_t kKeepBlocks = 64;
std::mutex blocks_mutex;
std::vector<Block> live_blocks, kept_blocks;

void free_block(const Block& b) {
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != b.device) cudaSetDevice(b.device);
    if (cudaFree(b.p) != cudaSuccess) cudaGetLastError();
    if (cur != b.device) cudaSetDevice(cur);
}

void free_kept_locked() {
    for (const Block& b : kept_blocks) free_block(b);
    kept_blocks.clear();
}
}  // namespace

void release_kept_blocks() {
    std::lock_guard<std::mutex> lock(blocks_mutex);
    free_kept_locked();
}

void dev_alloc(void** p, size_t bytes) {
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    int device = 0;
    if (!cuda_ok(cudaGetDevice(&device), "cudaGetDevice")) return;
    std::lock_guard<std::mutex> lock(blocks_mutex);
    // the smallest kept block that holds the request without wasting more than half of itself
    int best = -1;
    for (int k = 0; k < (int)kept_blocks.size(); ++k) {
        const Block& b = kept_blocks[k];
        if (b.device == device && b.bytes >= bytes && b.bytes <= 2 * bytes + 4096 &&
            (best < 0 || b.bytes < kept_blocks[best].bytes))
            best = k;
    }
    if (best >= 0 && !kept_blocks[best].idle) {
        if (cuda_ok(cudaDeviceSynchronize(), "cudaDeviceSynchronize")) {
            for (Block& b : kept_blocks)
                if (b.device == device) b.idle = true;
        } else {
            best = -1;
        }
    }
    if (best >= 0) {
        live_blocks.push_back(kept_blocks[best]);
        kept_blocks.erase(kept_blocks.begin() + best);
        *p = live_blocks.back().p;
    } else {
        cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation && !kept_blocks.empty()) {
            cudaGetLastError();
            free_kept_locked();
            e = cudaMalloc(p, bytes);
        }
        if (!cuda_ok(e, "cudaMalloc")) {
            *p = nullptr;
            return;
        }
        live_blocks.push_back(Block{*p, bytes, device, false});
    }
    g_state.dev_bytes += (long long)bytes;
}

void dev_free(void** p) {
    if (!*p) return;
    std::lock_guard<std::mutex> lock(blocks_mutex);
    for (size_t k = 0; k < live_blocks.size(); ++k) {
        if (live_blocks[k].p != *p) continue;
        Block b = live_blocks[k];
        b.idle = false;
        live_blocks.erase(live_blocks.begin() + k);
        // room for it: the longest-kept blocks go back to the device first
        size_t total = b.bytes;
        for (const Block& q : kept_blocks) total += q.bytes;
        while (!kept_blocks.empty() && (total > kKeepBytes || kept_blocks.size() >= kKeepBlocks)) {
            total -= kept_blocks.front().bytes;
            free_block(kept_blocks.front());
            kept_blocks.erase(kept_blocks.begin());
        }
        if (total <= kKeepBytes) kept_blocks.push_back(b);
        else free_block(b);
        break;
    }
    *p = nullptr;
}

const char* kernel_name(int id) {
    static const char* names[K_COUNT] = {"force_lj", "force_dem", "integrate", "ghost_sync", "final_integrate",
                                         "enforce_pbc", "borders", "binning", "neighbor_list", "scan", "reduce",
                                         "adjoint_hvp", "adjoint_step", "misc"};
    return (id >= 0 && id < K_COUNT) ? names[id] : "?";
}

// ---------------------------------------------------------------------------
// GPU phase timeline (CUDA events at phase changes on the library stream)
// ---------------------------------------------------------------------------
namespace {
struct Mark {
    cudaEvent_t ev;
    int phase;
};
std::vector<cudaEvent_t> ev_pool;
std::deque<Mark> marks;
double phase_ms[PH_COUNT] = {0};
int cur_phase = 0;

struct ProfRec {
    cudaEvent_t a, b;
    int k;
};
std::deque<ProfRec> prof_q;
long long prof_launch[K_COUNT] = {0};
double prof_ms[K_COUNT] = {0};
int prof_mask = 0;
int prof_every = 1;
long long prof_seen[K_COUNT] = {0};
cudaEvent_t prof_open[K_COUNT] = {nullptr};

cudaEvent_t get_event() {
    if (!ev_pool.empty()) {
        cudaEvent_t e = ev_pool.back();
        ev_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    TMD_CUDA(cudaEventCreate(&e));
    return e;
}
void put_event(cudaEvent_t e) { ev_pool.push_back(e); }

void fold_marks(bool all) {
    while (marks.size() >= 2) {
        const Mark& a = marks[0];
        const Mark& b = marks[1];
        if (!all && cudaEventQuery(b.ev) != cudaSuccess) break;
        if (all) cudaEventSynchronize(b.ev);
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, a.ev, b.ev) == cudaSuccess && a.phase > 0 && a.phase < PH_COUNT)
            phase_ms[a.phase] += ms;
        put_event(a.ev);
        marks.pop_front();
    }
}

void fold_prof(bool all) {
    while (!prof_q.empty()) {
        ProfRec& r = prof_q.front();
        if (!all && cudaEventQuery(r.b) != cudaSuccess) break;
        if (all) cudaEventSynchronize(r.b);
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, r.a, r.b) == cudaSuccess) {
            prof_ms[r.k] += ms;
            prof_launch[r.k]++;
        }
        put_event(r.a);
        put_event(r.b);
        prof_q.pop_front();
    }
}
}  // namespace

// device phase timing (md_get_phase_times) is opt-in: each mark is a timing event, and an
// event on the stream costs a few microseconds of pipeline drain
bool phase_on = false;

void phase_mark(int phase) {
    if (!phase_on || phase == cur_phase) return;
    cudaEvent_t e = get_event();
    TMD_CUDA(cudaEventRecord(e, g_state.stream));
    marks.push_back({e, phase});
    cur_phase = phase;
    if (marks.size() > 512) fold_marks(false);
}

void phase_times(double* out6) {
    if (phase_on) {
        cudaEvent_t e = get_event();
        TMD_CUDA(cudaEventRecord(e, g_state.stream));
        marks.push_back({e, cur_phase});
    }
    fold_marks(true);
    double tot = 0;
    for (int p = 1; p < PH_COUNT; ++p) tot += phase_ms[p];
    out6[0] = tot;
    out6[1] = phase_ms[PH_FORCE];
    out6[2] = phase_ms[PH_NEIGH];
    out6[3] = phase_ms[PH_COMM];
    out6[4] = phase_ms[PH_BALANCE];
    out6[5] = phase_ms[PH_OTHER];
}

void phase_reset() {
    fold_marks(true);
    for (auto& m : marks) put_event(m.ev);
    marks.clear();
    for (double& v : phase_ms) v = 0;
    cur_phase = 0;
}

void prof_begin(int k) {
    if (!(prof_mask & (1 << k))) return;
    if (prof_seen[k]++ % prof_every != 0) return;  // one launch in prof_every is timed
    prof_open[k] = get_event();
    TMD_CUDA(cudaEventRecord(prof_open[k], g_state.stream));
}

void prof_end(int k) {
    if (!(prof_mask & (1 << k)) || !prof_open[k]) return;
    cudaEvent_t b = get_event();
    TMD_CUDA(cudaEventRecord(b, g_state.stream));
    prof_q.push_back({prof_open[k], b, k});
    prof_open[k] = nullptr;
    if (prof_q.size() > 512) fold_prof(false);
}

void prof_reset() {
    fold_prof(true);
    for (int k = 0; k < K_COUNT; ++k) {
        prof_launch[k] = 0;
        prof_ms[k] = 0;
        prof_seen[k] = 0;
    }
}

// ---------------------------------------------------------------------------
// allocation
// ---------------------------------------------------------------------------
namespace {

// The per-slot arrays live in one device allocation per capacity: a few dozen allocations of a
// few MB each took ~11 ms to make and ~9 ms to free on B200, one allocation of their total
// size ~0.4 ms.  `elems` are the elements per slot, `keep` whether a growth copies the contents.
struct SlabItem {
    void** p;
    size_t elem, elems;
    bool keep;
};

template <class T>
SlabItem item(T** p, size_t elems, bool keep) {
    return SlabItem{reinterpret_cast<void**>(p), sizeof(T), elems, keep};
}

std::vector<SlabItem> slab_items(State& s) {
    std::vector<SlabItem> v;
    for (int b = 0; b < 2; ++b) {
        v.push_back(item(&s.pos.b[b], 1, true));
        v.push_back(item(&s.vel.b[b], 1, true));
        v.push_back(item(&s.frc.b[b], 1, true));
        v.push_back(item(&s.mass.b[b], 1, true));
        v.push_back(item(&s.ref.b[b], 1, true));
        v.push_back(item(&s.img.b[b], 1, true));
        v.push_back(item(&s.pos32.b[b], 1, true));
    }
    v.push_back(item(&s.frc32, 1, true));
    int** keep[] = {&s.rbk, &s.slot_of_ref, &s.rref, &s.gsrc, &s.groot, &s.gcode, &s.bsrc_ref, &s.broot_ref,
                    &s.bcode};
    for (int** q : keep) v.push_back(item(q, 1, true));
    int** scratch[] = {&s.bin_cell, &s.bin_rank, &s.tmp_key, &s.tmp_src, &s.nbn, &s.slot_cell, &s.chain};
    for (int** q : scratch) v.push_back(item(q, 1, false));
    v.push_back(item(&s.img_cnt, 2, false));
    v.push_back(item(&s.img_slot, kImgW, false));
    v.push_back(item(&s.dl_buf, 10, false));  // host-mirror transfers: mass, pos[3], vel[3], frc[3]
    return v;
}

// the events of a grid
void free_sync_objects(State& s) {
    for (cudaEvent_t& e : s.thermo_ev) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    s.sync_device = -1;
}

void free_all(State& s) {
    for (SlabItem& it : slab_items(s)) *it.p = nullptr;  // carved from the slab, freed with it
    dfree(&s.slab);
    int** ip[] = {&s.cnt, &s.cstart, &s.bcount, &s.scan_part};
    for (int** q : ip) dfree(q);
    dfree(&s.lb_tiles);
    s.lb_tile_cap = 0;
    s.img_ok = 0;
    s.ghosts_pushed = 0;
    dfree(&s.bmask);
    dfree(&s.nbl);
    dfree(&s.red_part);
    // the events stay for the next grid (made anew when the device changes)
    if (s.status_pending) await_words(s, &s.status_host->build, kStatusWords);
    s.status_pending = false;
    for (int k = 0; k < kThermoSlots; ++k) s.thermo_slot_ticket[k] = -1;
    dfree(&s.thermo_dev);
    dfree(&s.status_dev);
    s.scan_part_cap = 0;
    s.red_part_cap = 0;
    s.red_q0 = s.red_q1 = 0;
    s.dev_bytes = 0;
}

}  // namespace

// grows every per-slot array to hold `need` slots, keeping contents; false (error latched,
// arrays unchanged) when the device has no room
bool grow_atoms(State& s, int need) {
    if (s.mirror_pending) materialize_mirror(s);  // dl_buf is carved from the slab
    const int oldc = s.capA;
    // a multiple of 64 slots: per-slot planes laid out back to back (img_slot) start on
    // 256-byte boundaries, as bulk prefetches need
    const int newc = (need + need / 10 + 1024 + 63) & ~63;
    const size_t o = (size_t)oldc, n = (size_t)newc;
    std::vector<SlabItem> items = slab_items(s);
    size_t total = 0;
    for (const SlabItem& it : items) total += (it.elem * it.elems * n + 255) & ~(size_t)255;
    char* slab = nullptr;
    dalloc(&slab, total);
    if (!slab) return false;
    size_t off = 0;
    for (SlabItem& it : items) {
        char* q = slab + off;
        off += (it.elem * it.elems * n + 255) & ~(size_t)255;
        if (it.keep && *it.p && o)
            TMD_CUDA(cudaMemcpyAsync(q, *it.p, it.elem * it.elems * std::min(o, n), cudaMemcpyDeviceToDevice,
                                     s.stream));
        *it.p = q;
    }
    if (s.slab) {
        TMD_CUDA(cudaStreamSynchronize(s.stream));  // the copies out of the old slab
        dfree(&s.slab);
    }
    s.slab = slab;
    s.img_ok = 0;
    s.capA = newc;
    if (oldc > 0) std::printf("%d> reallocate_particle_capacity(): %d\n", comm().rank(), newc);
    return true;
}

// list capacity in entries per atom, a multiple of four (the list is stored in quads)
int list_rows(int rows) { return (std::max(rows, 4) + 3) & ~3; }
// entries allocated for the lists: one quad row more than the capacity, which the mixed force
// kernels read ahead into after an atom's last quad (the row is never used)
size_t list_entries(const State& s) { return (size_t)(s.nb_cap + 4) * s.nb_stride; }

void grow_lists(State& s, int rows) {
    dfree(&s.nbl);
    s.nb_cap = list_rows(rows);
    s.two_short = false;
    dalloc(&s.nbl, list_entries(s));
    s.lists_valid = 0;
}

// A rank's local count changes when atoms migrate: the border masks and counts and the list
// stride follow it (contents are not kept: every user writes them anew after a migration).
bool ensure_locals(State& s, int n) {
    n = std::max(n, 1);
    const int nblk = border_blocks(n);
    if (n > s.nb_stride) {
        s.nb_stride = ((n + n / 8 + 31) / 32) * 32;
        dfree(&s.nbl);
        dalloc(&s.nbl, list_entries(s));
        dfree(&s.bmask);
        dalloc(&s.bmask, (size_t)s.nb_stride);
        dfree(&s.bcount);
        dalloc(&s.bcount, (size_t)2 * 27 * border_blocks(s.nb_stride) + 1);
        s.lists_valid = 0;
    }
    ensure_scan_scratch(s, 27 * nblk);
    return s.nbl && s.bmask && s.bcount;
}

namespace {

bool allocate_state(State& s, int N, int nb_cap) {
    s.capA = 0;
    if (!grow_atoms(s, N + N / 2 + 64)) return false;
    const int ncells = s.geo.ncells;
    const int nseg = 2 * (ncells + 1);
    dalloc(&s.cnt, nseg + 1);
    dalloc(&s.cstart, nseg + 1);
    // sized by the list stride (at least N), which ensure_locals grows with the local count
    s.nb_stride = ((std::max(N, 1) + 31) / 32) * 32;
    dalloc(&s.bmask, (size_t)s.nb_stride);
    const int nblk = border_blocks(s.nb_stride);
    dalloc(&s.bcount, (size_t)2 * 27 * nblk + 1);  // border types (26) or migration classes (27), scanned
    s.nb_cap = list_rows(nb_cap > 0 ? nb_cap : 100);
    dalloc(&s.nbl, list_entries(s));
    if (s.sync_device != s.device) {
        free_sync_objects(s);
        for (int k = 0; k < kThermoSlots; ++k)
            TMD_CUDA(cudaEventCreateWithFlags(&s.thermo_ev[k], cudaEventDisableTiming));
        s.sync_device = s.device;
    }
    dalloc(&s.thermo_dev, 8);
    dalloc(&s.status_dev, 1);
    if (!s.status_host) TMD_CUDA(cudaMallocHost((void**)&s.status_host, sizeof(HostStatus)));
    if (!s.thermo_host) TMD_CUDA(cudaMallocHost((void**)&s.thermo_host, kThermoSlots * 4 * sizeof(double)));
    for (int k = 0; k < kThermoSlots; ++k) s.thermo_slot_ticket[k] = -1;
    s.thermo_tickets = 0;
    TMD_CUDA(cudaMemsetAsync(s.status_dev, 0, sizeof(DevStatus), s.stream));
    TMD_CUDA(cudaMemsetAsync(s.thermo_dev, 0, 8 * sizeof(double), s.stream));
    ensure_scan_scratch(s, std::max(nseg, 26 * nblk));
    return s.cnt && s.cstart && s.bmask && s.bcount && s.nbl && s.thermo_dev && s.status_dev;
}

bool require_alive(const char* what) {
    if (!g_state.alive) {
        set_error(MD_ERR_STATE, std::string(what) + " called before md_initialize_grid");
        return false;
    }
    return true;
}

// ---------------------------------------------------------------------------
// deferred work
// ---------------------------------------------------------------------------
void launch_force(State& s, const PendingForce& p, bool fuse_final, double dt) {
    resolve_lists(s);
    if (!p.half || p.dem || s.precision == 1) one_sided_lists(s);
    s.last_force_half = p.half ? 1 : 0;
    if (p.dem) run_force_dem(s, p);
    else run_force_lj(s, p, fuse_final, dt);
}

// the held-back final kick joins the integration when one is pending (same arithmetic)
double take_kick(State& s) {
    if (!s.pend_kick) return -1.0;
    s.pend_kick = false;
    return s.pend_kick_dt;
}

void flush_init(State& s) {
    if (!s.pend_init) return;
    s.pend_init = false;
    phase_mark(PH_FORCE);
    run_integrate(s, s.pend_dt, false, take_kick(s));
}

void flush_kick(State& s) {
    if (!s.pend_kick) return;
    s.pend_kick = false;
    phase_mark(PH_FORCE);
    run_final(s, s.pend_kick_dt);
}

void flush_force(State& s) {
    if (!s.pend_force.valid) return;
    PendingForce p = s.pend_force;
    s.pend_force.valid = false;
    phase_mark(PH_FORCE);
    launch_force(s, p, false, 0.0);
}

// a force held back by md_final_integration: launched with its final kick alone
void flush_final(State& s) {
    if (!s.pend_final) return;
    s.pend_final = false;
    phase_mark(PH_FORCE);
    launch_force(s, s.final_cfg, true, s.pend_final_dt);
}

// ghosts after a fused force + initial integration, when no ghost refresh follows: carried
// over as the unfused initial integration does
void flush_ghost(State& s) {
    if (!s.pend_ghost) return;
    s.pend_ghost = false;
    phase_mark(PH_FORCE);
    run_ghost_refresh(s, 0);
}

void flush_pbc(State& s) {
    if (!s.pend_pbc) return;
    s.pend_pbc = false;
    phase_mark(PH_OTHER);
    run_enforce_pbc(s);
}

// resolve: complete a deferred list build even when nothing else is pending (calls that read
// the host-side state); md_compute_* only queue a force and skip that
void flush_all(State& s, bool resolve = true) {
    if (resolve || s.pend_links || s.pend_final || s.pend_ghost || s.pend_init || s.pend_kick ||
        s.pend_force.valid || s.pend_pbc)
        resolve_lists(s);
    flush_links(s);
    flush_final(s);
    flush_ghost(s);
    flush_init(s);
    flush_kick(s);
    flush_force(s);
    flush_pbc(s);
}

// everything but the carried-over ghosts: for calls that touch only the locals, so that a
// following md_borders, which writes every ghost anew, can drop the carry
void flush_locals(State& s) {
    resolve_lists(s);
    flush_links(s);
    flush_final(s);
    flush_init(s);
    flush_kick(s);
    flush_force(s);
    flush_pbc(s);
}

void sync_stream(State& s) { TMD_CUDA(cudaStreamSynchronize(s.stream)); }

// device state -> the host mirror's layout, by reference index r (a permutation of the slots):
// out = mass[NA], pos[NA][3], vel[NA][3], frc[NA][3]; ghost velocities only for the
// contact-fixed DEM model, ghost forces zero (what md_copy_data_from_accelerator reports)
__global__ void k_gather_ref(const double4* __restrict__ pos, const double4* __restrict__ vel,
                             const double4* __restrict__ frc, const float4* __restrict__ frc32,
                             const double* __restrict__ mass, const int* __restrict__ ref, double* __restrict__ out,
                             int N, int NA, int mixed, int ghost_vel) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int slot = blk * blockDim.x + threadIdx.x;
    if (slot >= NA) return;
    const int r = ref[slot];
    if (r < 0 || r >= NA) return;
    double* om = out;
    double* op = out + NA;
    double* ov = out + 4 * (size_t)NA;
    double* of = out + 7 * (size_t)NA;
    om[r] = mass[slot];
    const double4 p = ldg_d4(pos + slot);
    op[3 * (size_t)r] = p.x;
    op[3 * (size_t)r + 1] = p.y;
    op[3 * (size_t)r + 2] = p.z;
    double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
    if (r < N || ghost_vel) v = ldg_d4(vel + slot);
    ov[3 * (size_t)r] = v.x;
    ov[3 * (size_t)r + 1] = v.y;
    ov[3 * (size_t)r + 2] = v.z;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (r < N) {
        if (mixed) {
            const float4 f = frc32[slot];
            fx = f.x, fy = f.y, fz = f.z;
        } else {
            const double4 f = ldg_d4(frc + slot);
            fx = f.x, fy = f.y, fz = f.z;
        }
    }
    of[3 * (size_t)r] = fx;
    of[3 * (size_t)r + 1] = fy;
    of[3 * (size_t)r + 2] = fz;
}

// host mirror (input order: mass[n], pos[n][3], vel[n][3]) -> slot arrays, slot = reference
// index; forces zero, no wraps yet
__global__ void k_upload(const double* __restrict__ m, const double* __restrict__ p, const double* __restrict__ v,
                         double4* __restrict__ pos, double4* __restrict__ vel, double4* __restrict__ frc,
                         float4* __restrict__ frc32, double* __restrict__ mass, int* __restrict__ ref,
                         int* __restrict__ slot_of_ref, int* __restrict__ img, int n) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t k = 3 * (size_t)i;
    st_d4(pos + i, make_double4(p[k], p[k + 1], p[k + 2], 0.0));
    st_d4(vel + i, make_double4(v[k], v[k + 1], v[k + 2], 0.0));
    st_d4(frc + i, make_double4(0.0, 0.0, 0.0, 0.0));
    frc32[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    mass[i] = m[i];
    ref[i] = i;
    slot_of_ref[i] = i;
    img[i] = 0;
}

__global__ void k_convert_forces(double4* f64, float4* f32, int n, int to32) {
    const int blk = (int)blockIdx.x + pdl_wait();
    int i = blk * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (to32) {
        double4 f = f64[i];
        f32[i] = make_float4((float)f.x, (float)f.y, (float)f.z, 0.f);
    } else {
        float4 f = f32[i];
        f64[i] = make_double4(f.x, f.y, f.z, 0.0);
    }
}

// downloads slot data and scatters it to reference order
struct Snapshot {
    std::vector<double4> pos, vel, frc;
    std::vector<float4> frc32;
    std::vector<double> mass;
    std::vector<int> ref;
};

void snapshot(State& s, Snapshot& sn) {
    flush_all(s);
    const int NA = s.N + s.G;
    sn.pos.resize(NA);
    sn.vel.resize(NA);
    sn.frc.resize(NA);
    sn.frc32.resize(NA);
    sn.mass.resize(NA);
    sn.ref.resize(NA);
    if (NA == 0) return;
    TMD_CUDA(cudaMemcpyAsync(sn.pos.data(), s.pos.b[s.pc], sizeof(double4) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(sn.vel.data(), s.vel.b[s.vc], sizeof(double4) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(sn.frc.data(), s.frc.b[s.ac], sizeof(double4) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(sn.frc32.data(), s.frc32, sizeof(float4) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(sn.mass.data(), s.mass.b[s.ac], sizeof(double) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(sn.ref.data(), s.ref.b[s.ac], sizeof(int) * NA, cudaMemcpyDeviceToHost, s.stream));
    sync_stream(s);
}

// std::cout default formatting of a double (6 significant digits)
void print_g(double v) { std::printf("%g", v); }

double host_temperature(const State& s) {  // core/thermo.impala:1-16 on the host mirror
    const double mass = 1.0, mvv2e = 1.0;
    int dof = s.N * 3 - 3;
    double t_scale = mvv2e / (double)dof;
    double t = 0.0;
    for (int i = 0; i < s.N; ++i) {
        const double* v = &s.h_vel[(size_t)i * 3];
        t += (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * mass;
    }
    return t * t_scale;
}

}  // namespace

// copies of the snapshot in dl_buf ([mass NA][pos 3NA][vel 3NA][frc 3NA], reference order):
// rows [r0, r1) of each array into the given destinations
static void copy_snapshot(State& s, int r0, int r1, double* m, double* x, double* v, double* f) {
    const size_t na = (size_t)s.mirror_na, a = (size_t)r0, n = (size_t)(r1 - r0);
    if (n == 0) return;
    TMD_CUDA(cudaMemcpyAsync(m, s.dl_buf + a, sizeof(double) * n, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(x, s.dl_buf + na + 3 * a, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(v, s.dl_buf + 4 * na + 3 * a, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost,
                             s.stream));
    TMD_CUDA(cudaMemcpyAsync(f, s.dl_buf + 7 * na + 3 * a, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost,
                             s.stream));
}

void materialize_mirror(State& s, int parts) {
    const int todo = s.mirror_pending & parts;
    if (!todo) return;
    const int n = s.mirror_n, na = s.mirror_na;
    if ((todo & 1) && s.x0_in_pos) {  // the initial positions are about to be overwritten
        s.h_x0.assign(s.h_pos.begin(), s.h_pos.begin() + 3 * (size_t)n);
        s.x0_in_pos = false;
    }
    if (todo & 1) s.mirror_frc_zero = false;
    if (todo & 1) copy_snapshot(s, 0, n, s.h_mass.data(), s.h_pos.data(), s.h_vel.data(), s.h_frc.data());
    if (todo & 2)
        copy_snapshot(s, n, na, s.h_mass.data() + n, s.h_pos.data() + 3 * (size_t)n, s.h_vel.data() + 3 * (size_t)n,
                      s.h_frc.data() + 3 * (size_t)n);
    TMD_CUDA(cudaStreamSynchronize(s.stream));
    s.mirror_pending &= ~todo;
}

}  // namespace tmd

using namespace tmd;

extern "C" {

// a list build whose status is still in flight may latch an error (locals outside the grid)
int md_last_error(void) {
    if (g_state.alive) resolve_lists(g_state);
    return g_state.last_error;
}
const char* md_last_error_string(void) {
    if (g_state.alive) resolve_lists(g_state);
    return g_state.last_error_msg.c_str();
}
void md_clear_error(void) {
    if (g_state.alive) resolve_lists(g_state);
    g_state.last_error = 0;
    g_state.last_error_msg.clear();
}

void md_set_stream(void* stream) {
    State& s = g_state;
    if (s.alive) flush_all(s);
    if (s.own_stream && s.stream) {
        cudaStreamSynchronize(s.stream);
        cudaStreamDestroy(s.stream);
    }
    s.stream = (cudaStream_t)stream;
    s.own_stream = false;
    s.stream_set = true;
}

// core/runtime.impala:7-37
int md_initialize_grid(double const* masses, Vector3D const* positions, Vector3D const* velocities, int n,
                       double const* aabb, double const* rank_aabb, double cell_spacing, int cell_capacity,
                       int neighborlist_capacity) {
    Range range("md_initialize_grid");
    (void)cell_capacity;  // cells are a counting sort here: no per-cell capacity
    State& s = g_state;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error(MD_ERR_NO_DEVICE, "no CUDA device available");
        return -1;
    }
    if (n < 0 || n >= kMaxSlots / 2 || !(cell_spacing > 0.0)) {
        set_error(MD_ERR_ARGUMENT, "md_initialize_grid: invalid particle count or cell spacing");
        return -1;
    }
    if (s.alive) md_deallocate_grid();
    Comm& cm = comm();
    if (cm.active()) {
        // several ranks: the layout of md_get_node_bounding_box (made here from the world box
        // when the caller skipped it); every divided axis must hold a full halo per rank
        if (!cm.topo_set || cm.topo.world != cm.world() || cm.topo.rank != cm.rank()) {
            double len[3];
            int dims[3];
            for (int d = 0; d < 3; ++d) len[d] = aabb[2 * d + 1] - aabb[2 * d];
            node_config(cm.world(), len, dims);
            make_topology(cm.world(), cm.rank(), dims, cm.topo);
            cm.topo_set = true;
        }
        for (int d = 0; d < 3; ++d)
            if (cm.topo.dims[d] > 1 && rank_aabb[2 * d + 1] - rank_aabb[2 * d] < cell_spacing) {
                set_error(MD_ERR_ARGUMENT, "md_initialize_grid: a rank box is narrower than the cell spacing "
                                           "(too many ranks for this box)");
                return -1;
            }
    }
    TMD_CUDA(cudaGetDevice(&s.device));
    if (!s.stream && !s.stream_set) {
        TMD_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
        s.own_stream = true;
    }
    Geometry& g = s.geo;
    for (int d = 0; d < 3; ++d) {
        g.world_lo[d] = aabb[2 * d];
        g.world_hi[d] = aabb[2 * d + 1];
        g.aabb_lo[d] = rank_aabb[2 * d] - cell_spacing;
        g.aabb_hi[d] = rank_aabb[2 * d + 1] + cell_spacing;
        g.len[d] = g.world_hi[d] - g.world_lo[d];
    }
    g.spacing = cell_spacing;
    // core/grid.impala:94-98
    g.nx = (int)std::floor((g.aabb_hi[0] - g.aabb_lo[0] + (cell_spacing / 2.0)) / cell_spacing) + 1;
    g.ny = (int)std::floor((g.aabb_hi[1] - g.aabb_lo[1] + (cell_spacing / 2.0)) / cell_spacing) + 1;
    g.nz = (int)std::floor((g.aabb_hi[2] - g.aabb_lo[2] + (cell_spacing / 2.0)) / cell_spacing) + 1;
    g.ncells = g.nx * g.ny * g.nz;
    // dyadic rebasing grid strictly wider than the cell spacing (mixed form)
    g.rb_h = (std::floor(cell_spacing * 8.0) + 1.0) / 8.0;

    s.N = n;
    s.G = 0;
    s.halo.on = cm.active();
    if (s.halo.on) s.ghost_exact = 1;  // ghosts of other ranks are exact images; own ones likewise
    s.pc = s.vc = s.ac = 0;
    s.lists_valid = 0;
    s.lists_two = s.two_short = false;
    s.force_seen = false;
    s.cells_filled = 0;
    s.pend_init = false;
    s.pend_force = PendingForce();
    s.pend_final = s.pend_ghost = s.pend_kick = s.pend_pbc = false;
    s.bin_zeroed = s.build_zeroed = s.pend_links = false;
    s.mirror_pending = 0;
    s.force_iters = s.rsq_iters = s.integration_iters = 0;
    s.launches = 0;
    if (!allocate_state(s, n, neighborlist_capacity)) {
        free_all(s);
        return -1;  // the error (a failed device allocation) is latched
    }

    // core/grid.impala:215-249: the host mirror in input order
    static_assert(sizeof(Vector3D) == 3 * sizeof(double), "Vector3D is three packed doubles");
    s.h_mass.resize(n);
    s.h_pos.resize((size_t)n * 3);
    s.h_vel.resize((size_t)n * 3);
    s.h_frc.resize((size_t)n * 3);
    if (n > 0) {
        std::memcpy(s.h_mass.data(), masses, sizeof(double) * n);
        std::memcpy(s.h_pos.data(), positions, sizeof(Vector3D) * n);
        std::memcpy(s.h_vel.data(), velocities, sizeof(Vector3D) * n);
    }
    // the mirror's forces are zero (written out as zeros until a snapshot fills them) and the
    // initial positions are the mirror's until a snapshot overwrites them (kept aside then)
    s.mirror_frc_zero = true;
    s.x0_in_pos = true;
    s.alive = true;
    phase_reset();
    return s.N;
}

// core/runtime.impala:158-186 (host mirror, sequential sums as the reference)
void md_create_velocity(double t_request) {
    State& s = g_state;
    if (!require_alive("md_create_velocity")) return;
    materialize_mirror(s);
    const int n = s.N;
    Comm& cm = comm();
    long long ntot = n;
    double vt[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < n; ++i)
        for (int d = 0; d < 3; ++d) vt[d] = vt[d] + s.h_vel[3 * i + d];
    if (cm.active() && !(cm.allreduce_sum(&ntot, 1) && cm.allreduce_sum(vt, 3))) {
        set_error(MD_ERR_COMM, "md_create_velocity: " + cm.error());
        return;
    }
    for (int d = 0; d < 3; ++d) vt[d] = vt[d] / (double)ntot;
    // the mean removed and core/thermo.impala:1-16's sum taken in the same pass (same terms in
    // the same order as a separate pass over the updated velocities)
    double t = 0.0;
    for (int i = 0; i < n; ++i) {
        double* v = &s.h_vel[(size_t)i * 3];
        for (int d = 0; d < 3; ++d) v[d] = v[d] - vt[d];
        t += (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * 1.0;
    }
    if (cm.active() && !cm.allreduce_sum(&t, 1)) {
        set_error(MD_ERR_COMM, "md_create_velocity: " + cm.error());
        return;
    }
    t = t * (1.0 / (double)(ntot * 3 - 3));
    double factor = std::sqrt(t_request / t);
    for (int i = 0; i < n; ++i)
        for (int d = 0; d < 3; ++d) s.h_vel[3 * i + d] = s.h_vel[3 * i + d] * factor;
}

// core/grid.impala:360-367
void md_copy_data_to_accelerator(void) {
    Range range("md_copy_data_to_accelerator");
    State& s = g_state;
    if (!require_alive("md_copy_data_to_accelerator")) return;
    flush_all(s);
    materialize_mirror(s);  // the upload goes through dl_buf
    const int N = s.N;
    s.G = 0;
    s.pc = s.vc = s.ac = 0;
    if (N == 0) return;
    // the mirror (page-locked, reference order = input order here) goes up as it is and is
    // spread into the slot arrays on the device
    double* dm = s.dl_buf;
    double* dp = s.dl_buf + N;
    double* dv = s.dl_buf + 4 * (size_t)N;
    TMD_CUDA(cudaMemcpyAsync(dm, s.h_mass.data(), sizeof(double) * N, cudaMemcpyHostToDevice, s.stream));
    TMD_CUDA(cudaMemcpyAsync(dp, s.h_pos.data(), sizeof(double) * 3 * N, cudaMemcpyHostToDevice, s.stream));
    TMD_CUDA(cudaMemcpyAsync(dv, s.h_vel.data(), sizeof(double) * 3 * N, cudaMemcpyHostToDevice, s.stream));
    launch(s, (N + 255) / 256, 256, 0, k_upload, dm, dp, dv, s.pos.b[0], s.vel.b[0], s.frc.b[0], s.frc32,
           s.mass.b[0], s.ref.b[0], s.slot_of_ref, s.img.b[0], N);
    launched(K_MISC);
    // the mirror may be resized (and moved) by later calls: wait for the copies out of it
    sync_stream(s);
}

// core/grid.impala:369-374: device -> host mirror, scattered to reference order.  The state is
// gathered into reference order on the device now (the snapshot); the copy to the host happens
// when a reader needs it, and then only the part it needs: md_write_grid_data_to_arrays takes
// the locals straight into the caller's arrays.
void md_copy_data_from_accelerator(void) {
    Range range("md_copy_data_from_accelerator");
    State& s = g_state;
    if (!require_alive("md_copy_data_from_accelerator")) return;
    flush_all(s);
    const int NA = s.N + s.G;
    // every element is overwritten when the pending parts are copied (all NA reference indices)
    s.h_mass.resize(NA);
    s.h_pos.resize((size_t)NA * 3);
    s.h_vel.resize((size_t)NA * 3);
    s.h_frc.resize((size_t)NA * 3);
    s.mirror_pending = 0;
    if (NA == 0) return;
    launch(s, (NA + 255) / 256, 256, 0, k_gather_ref, s.pos.b[s.pc], s.vel.b[s.vc], s.frc.b[s.ac], s.frc32,
           s.mass.b[s.ac], s.ref.b[s.ac], s.dl_buf, s.N, NA, s.precision == 1, s.dem_fixed);
    launched(K_MISC);
    s.mirror_pending = (s.N > 0 ? 1 : 0) | (s.G > 0 ? 2 : 0);
    s.mirror_n = s.N;
    s.mirror_na = NA;
}

// comm/comm.impala:392-525: with one rank nothing leaves (the periodic wrap is md_enforce_pbc's);
// with several, locals beyond the rank box move to their new owner (k_halo.cu)
void md_exchange_particles(void) {
    Range range("md_exchange_particles");
    State& s = g_state;
    if (!require_alive("md_exchange_particles")) return;
    flush_locals(s);
    if (s.halo.on) {
        s.pend_ghost = false;  // every ghost is written anew by the border pass that follows
        phase_mark(PH_COMM);
        run_migrate(s);
    }
}

void md_enforce_pbc(void) {  // wraps locals only: a pending ghost carry stays pending
    Range range("md_enforce_pbc");
    State& s = g_state;
    if (!require_alive("md_enforce_pbc")) return;
    flush_locals(s);
    s.pend_pbc = true;  // held back for md_borders, which wraps in its first kernel
}

void md_borders(void) {
    Range range("md_borders");
    State& s = g_state;
    if (!require_alive("md_borders")) return;
    s.pend_ghost = false;  // every ghost is written anew below: the carry would be overwritten
    const bool wrap = s.pend_pbc;
    s.pend_pbc = false;
    flush_all(s);
    phase_mark(PH_COMM);
    run_borders(s, wrap);
}

void md_distribute_particles(void) {
    Range range("md_distribute_particles");
    State& s = g_state;
    if (!require_alive("md_distribute_particles")) return;
    flush_all(s);
    phase_mark(PH_OTHER);
    run_distribute(s);
}

void md_assemble_neighborlists(bool half, double cutoff) {
    Range range("md_assemble_neighborlists");
    State& s = g_state;
    if (!require_alive("md_assemble_neighborlists")) return;
    if (half && s.halo.on) {
        // a half list leaves the reaction on a ghost of another rank, which would need the
        // forces sent back: several ranks run full lists
        set_error(MD_ERR_UNSUPPORTED, "md_assemble_neighborlists: half lists on several ranks (use full lists)");
        return;
    }
    // pending ghost links stay pending when nothing else is (the list build then runs them as
    // extra blocks); any other pending work may read them, so then they go first, alone
    const bool hold = s.pend_links && !s.pend_force.valid && !s.pend_final && !s.pend_ghost && !s.pend_init &&
                      !s.pend_kick;
    if (hold) s.pend_links = false;
    flush_all(s);
    if (hold) s.pend_links = true;
    phase_mark(PH_NEIGH);
    run_build_lists(s, half, cutoff, true);
}

void md_initial_integration(double dt) {
    Range range("md_initial_integration");
    State& s = g_state;
    if (!require_alive("md_initial_integration")) return;
    if (s.pend_final && !s.pend_ghost && !s.pend_init && !s.pend_force.valid) {
        // the held-back force, its final kick and this initial integration in one kernel
        s.pend_final = false;
        phase_mark(PH_FORCE);
        run_force_lj_init(s, s.final_cfg, s.pend_final_dt, dt);
        s.pend_ghost = true;
        return;
    }
    if (s.pend_kick && !s.pend_final && !s.pend_ghost && !s.pend_init && !s.pend_force.valid) {
        s.pend_init = true;  // the held-back kick stays pending and joins this integration
        s.pend_dt = dt;
        return;
    }
    flush_all(s);
    s.pend_init = true;
    s.pend_dt = dt;
}

void md_synchronize_ghost_layer(void) {
    Range range("md_synchronize_ghost_layer");
    State& s = g_state;
    if (!require_alive("md_synchronize_ghost_layer")) return;
    resolve_lists(s);
    flush_links(s);
    flush_pbc(s);  // ghosts are refreshed from the wrapped locals
    flush_final(s);
    if (!s.pend_init) flush_kick(s);
    flush_force(s);
    // phase marks are timing events: set only where work is enqueued (an event on the
    // stream costs a few microseconds of pipeline drain)
    if (s.pend_ghost) {  // the fused kernel wrote the locals, and the ghosts if it could
        s.pend_ghost = false;
        const int gm = s.ghost_exact ? 2 : 1;
        if (s.ghosts_pushed != gm) {
            phase_mark(PH_COMM);
            run_ghost_refresh(s, gm);
        }
    } else if (s.pend_init) {
        s.pend_init = false;
        phase_mark(PH_COMM);
        run_integrate(s, s.pend_dt, true, take_kick(s));
    } else {
        phase_mark(PH_COMM);
        run_ghost_sync(s);
    }
    if (s.halo.on) {
        phase_mark(PH_COMM);
        run_halo_sync(s);
    }
}

void md_compute_lennard_jones(bool half, double rc, double eps, double sigma) {
    Range range("md_compute_lennard_jones");
    State& s = g_state;
    if (!require_alive("md_compute_lennard_jones")) return;
    flush_all(s, false);
    PendingForce p;
    p.valid = true;
    p.dem = false;
    p.half = half;
    p.rc = rc;
    p.eps = eps;
    p.sigma = sigma;
    s.pend_force = p;
    s.force_cfg = p;
    s.force_seen = true;
    s.last_rc = rc;
    s.last_eps = eps;
    s.last_sigma = sigma;
}

void md_compute_dem(bool half, double rc, double damping_n, double damping_t, double stiffness, double friction) {
    Range range("md_compute_dem");
    State& s = g_state;
    if (!require_alive("md_compute_dem")) return;
    flush_all(s, false);
    PendingForce p;
    p.valid = true;
    p.dem = true;
    p.half = half;
    p.rc = rc;
    p.dn = damping_n;
    p.dt_ = damping_t;
    p.k = stiffness;
    p.mu = friction;
    s.pend_force = p;
    s.force_cfg = p;
    s.force_seen = true;
}

void md_final_integration(double dt) {
    Range range("md_final_integration");
    State& s = g_state;
    if (!require_alive("md_final_integration")) return;
    flush_links(s);
    flush_pbc(s);
    flush_final(s);
    flush_ghost(s);
    flush_init(s);
    flush_kick(s);
    if (s.pend_force.valid) {
        PendingForce p = s.pend_force;
        s.pend_force.valid = false;
        if (force_init_fusable(s, p)) {
            // held back: the next md_initial_integration joins it (one pass over the atoms),
            // any other call launches it with this kick alone
            s.pend_final = true;
            s.pend_final_dt = dt;
            s.final_cfg = p;
            s.last_force_half = 0;
            return;
        }
        phase_mark(PH_FORCE);
        if (!p.dem && !p.half) {
            launch_force(s, p, true, dt);
            return;
        }
        launch_force(s, p, false, 0.0);
        if (!s.thermo) {
            // held back: the next initial integration applies it first (one launch fewer); the
            // thermo sums take their kinetic energy from the separate kick, so not with thermo
            s.pend_kick = true;
            s.pend_kick_dt = dt;
            return;
        }
    }
    phase_mark(PH_FORCE);
    run_final(s, dt);
}

// core/grid.impala:483-499 (host mirror)
int md_write_grid_data_to_arrays(double* m, Vector3D* x, Vector3D* v, Vector3D* f) {
    State& s = g_state;
    if (!require_alive("md_write_grid_data_to_arrays")) return 0;
    flush_all(s);
    if ((s.mirror_pending & 1) && s.mirror_n == s.N) {  // the snapshot's locals, straight to the caller
        copy_snapshot(s, 0, s.N, m, reinterpret_cast<double*>(x), reinterpret_cast<double*>(v),
                      reinterpret_cast<double*>(f));
        TMD_CUDA(cudaStreamSynchronize(s.stream));
        return s.N;
    }
    materialize_mirror(s);
    const size_t n = std::min((size_t)s.N, s.h_mass.size());
    if (n > 0) {
        std::memcpy(m, s.h_mass.data(), sizeof(double) * n);
        std::memcpy(x, s.h_pos.data(), sizeof(Vector3D) * n);
        std::memcpy(v, s.h_vel.data(), sizeof(Vector3D) * n);
        if (s.mirror_frc_zero) std::memset(f, 0, sizeof(Vector3D) * n);
        else std::memcpy(f, s.h_frc.data(), sizeof(Vector3D) * n);
    }
    return s.N;
}

// core/grid.impala:501-518: returns nparticles, as the reference does
int md_write_grid_ghost_data_to_arrays(double* m, Vector3D* x, Vector3D* v, Vector3D* f) {
    State& s = g_state;
    if (!require_alive("md_write_grid_ghost_data_to_arrays")) return 0;
    flush_all(s);
    if ((s.mirror_pending & 2) && s.mirror_n == s.N && s.mirror_na == s.N + s.G) {  // straight to the caller
        copy_snapshot(s, s.N, s.N + s.G, m, reinterpret_cast<double*>(x), reinterpret_cast<double*>(v),
                      reinterpret_cast<double*>(f));
        TMD_CUDA(cudaStreamSynchronize(s.stream));
        return s.N;
    }
    materialize_mirror(s);
    const size_t have = s.h_mass.size();
    const size_t n0 = (size_t)s.N;
    const size_t ng = have > n0 ? std::min((size_t)s.G, have - n0) : 0;
    if (ng > 0) {
        std::memcpy(m, s.h_mass.data() + n0, sizeof(double) * ng);
        std::memcpy(x, s.h_pos.data() + 3 * n0, sizeof(Vector3D) * ng);
        std::memcpy(v, s.h_vel.data() + 3 * n0, sizeof(Vector3D) * ng);
        std::memcpy(f, s.h_frc.data() + 3 * n0, sizeof(Vector3D) * ng);
    }
    return s.N;
}

// core/grid.impala:520-546
int md_write_grid_aabb_data_to_arrays(double* m, Vector3D* x, Vector3D* v, Vector3D* f) {
    State& s = g_state;
    const Geometry& g = s.geo;
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j)
            for (int k = 0; k < 2; ++k) {
                int idx = k * 4 + j * 2 + i;
                m[idx] = 0.0;
                x[idx] = Vector3D{i == 0 ? g.aabb_lo[0] : g.aabb_hi[0], j == 0 ? g.aabb_lo[1] : g.aabb_hi[1],
                                  k == 0 ? g.aabb_lo[2] : g.aabb_hi[2]};
                v[idx] = Vector3D{0.0, 0.0, 0.0};
                f[idx] = Vector3D{0.0, 0.0, 0.0};
            }
    return s.N;
}

void md_deallocate_grid(void) {
    State& s = g_state;
    if (s.alive) {
        flush_all(s);
        sync_stream(s);
    }
    fold_prof(true);
    phase_reset();
    free_all(s);
    halo_free(s);
    release_adjoint();
    s.mirror_pending = 0;
    s.alive = false;
    s.N = s.G = 0;
    s.capA = 0;
}

// core/runtime.impala:146-156 (host mirror)
void md_print_grid(void) {
    State& s = g_state;
    if (s.alive) materialize_mirror(s);
    for (int i = 0; i < s.N; ++i) {
        std::printf("0> pos_local: ");
        print_g(s.h_pos[3 * i]); std::printf(", "); print_g(s.h_pos[3 * i + 1]); std::printf(", ");
        print_g(s.h_pos[3 * i + 2]); std::printf("\n");
    }
    for (int i = 0; i < s.N; ++i) {
        std::printf("0> vel_local: ");
        print_g(s.h_vel[3 * i]); std::printf(", "); print_g(s.h_vel[3 * i + 1]); std::printf(", ");
        print_g(s.h_vel[3 * i + 2]); std::printf("\n");
    }
    std::fflush(stdout);
}

void md_print_ghost(void) {
    State& s = g_state;
    if (s.alive) materialize_mirror(s);
    const size_t have = s.h_mass.size();
    for (int i = s.N; i < s.N + s.G && (size_t)i < have; ++i) {
        std::printf("0> pos_ghost: ");
        print_g(s.h_pos[3 * i]); std::printf(", "); print_g(s.h_pos[3 * i + 1]); std::printf(", ");
        print_g(s.h_pos[3 * i + 2]); std::printf("\n");
    }
    for (int i = s.N; i < s.N + s.G && (size_t)i < have; ++i) {
        std::printf("0> vel_ghost: ");
        print_g(s.h_vel[3 * i]); std::printf(", "); print_g(s.h_vel[3 * i + 1]); std::printf(", ");
        print_g(s.h_vel[3 * i + 2]); std::printf("\n");
    }
    std::fflush(stdout);
}

// core/runtime.impala:250-251: the ranks of the environment connect (comm.cpp); one rank when
// the environment names none
void md_mpi_initialize(void) {
    if (!comm().init()) set_error(MD_ERR_COMM, "md_mpi_initialize: " + comm().error());
}
void md_mpi_finalize(void) {
    if (g_state.alive) md_deallocate_grid();
    free_sync_objects(g_state);
    release_kept_blocks();
    comm().finalize();
}
void md_barrier(void) {  // this rank's device work done, then every rank's
    State& s = g_state;
    if (s.alive) {
        flush_all(s);
        sync_stream(s);
    }
    if (comm().active() && !comm().barrier()) set_error(MD_ERR_COMM, "md_barrier: " + comm().error());
}
int md_get_world_size(void) { return comm().world(); }
int md_get_world_rank(void) { return comm().rank(); }
int md_get_number_of_particles(void) { return g_state.N; }
int md_get_number_of_ghost_particles(void) { return g_state.G; }

// comm/comm.impala:221-299: the rank layout that minimises the ranks' surface, this rank's
// place in the periodic cart and its box (one rank: the world box)
void md_get_node_bounding_box(double const* aabb, double (*rank)[6]) {
    Comm& cm = comm();
    double len[3];
    int dims[3];
    for (int d = 0; d < 3; ++d) len[d] = aabb[2 * d + 1] - aabb[2 * d];
    node_config(cm.world(), len, dims);
    make_topology(cm.world(), cm.rank(), dims, cm.topo);
    cm.topo_set = true;
    rank_box(aabb, dims, cm.topo.coords, *rank);
}

// load balancing / multi-process entry points (out of scope on one GPU)
void md_rescale_grid(double const* aabb) {
    (void)aabb;
    set_error(MD_ERR_UNSUPPORTED, "md_rescale_grid: load balancing is not supported on one GPU");
}
double md_get_send_buffer_value(int i) {
    (void)i;
    return 0.0;
}
void md_set_recv_buffer_value(int i, double v) {
    (void)i;
    (void)v;
}
void md_resize_recv_buffer_capacity(int c) { (void)c; }
int md_serialize_particles(double const* aabb) {
    (void)aabb;
    set_error(MD_ERR_UNSUPPORTED, "md_serialize_particles: load balancing is not supported on one GPU");
    return 0;
}
void md_deserialize_particles(int n) {
    (void)n;
    set_error(MD_ERR_UNSUPPORTED, "md_deserialize_particles: load balancing is not supported on one GPU");
}
void md_update_neighborhood(int nranks, int total, int const* ranks, int const* naabbs, double const* aabbs) {
    (void)nranks; (void)total; (void)ranks; (void)naabbs; (void)aabbs;
}

// core/runtime.impala:72-95: locals / ghosts inside the box
void md_compute_boundary_weights(double xmin, double xmax, double ymin, double ymax, double zmin, double zmax,
                                 unsigned long int* comp_w, unsigned long int* comm_w) {
    State& s = g_state;
    *comp_w = 0;
    *comm_w = 0;
    if (!s.alive) return;
    Snapshot sn;
    snapshot(s, sn);
    auto inside = [&](const double4& p) {
        return p.x >= xmin && p.x <= xmax && p.y >= ymin && p.y <= ymax && p.z >= zmin && p.z <= zmax;
    };
    for (int slot = 0; slot < s.N + s.G; ++slot) {
        if (!inside(sn.pos[slot])) continue;
        if (sn.ref[slot] < s.N) (*comp_w)++;
        else (*comm_w)++;
    }
}

// core/runtime.impala:280-296
void md_report_iterations(void) {
    State& s = g_state;
    long long total = 0;
    if (s.alive) {
        flush_all(s);
        one_sided_lists(s);
        std::vector<int> n(s.N);
        if (s.N) {
            TMD_CUDA(cudaMemcpyAsync(n.data(), s.nbn, sizeof(int) * s.N, cudaMemcpyDeviceToHost, s.stream));
            sync_stream(s);
        }
        if (s.lists_valid)
            for (int v : n) total += v;
        // pairs inside the cutoff of the last force call: its lists and positions are the
        // current ones (a step's last position update precedes its force)
        if (s.force_cfg.valid) s.rsq_iters = count_pairs_inside(s, s.force_cfg.rc);
    }
    s.force_iters = total;
    long long it[3] = {s.force_iters, s.rsq_iters, s.integration_iters};
    Comm& cm = comm();
    if (cm.active() && !cm.allreduce_sum(it, 3)) set_error(MD_ERR_COMM, "md_report_iterations: " + cm.error());
    if (cm.rank() != 0) return;  // the sums are printed once (core/runtime.impala:280-296)
    std::printf("ForceIters RsqIters IntegrationIters\n");
    std::printf("%lld %lld %lld \n", it[0], it[1], it[2]);
    std::fflush(stdout);
}

// core/runtime.impala:298-316 (temperature from the host mirror)
void md_report_particles(void) {
    State& s = g_state;
    if (s.alive) {
        flush_all(s);
        materialize_mirror(s, 1);
    }
    Comm& cm = comm();
    if (cm.active()) {  // sums over the ranks, printed once (core/runtime.impala:298-316)
        long long ng[2] = {s.N, s.G};
        double t = 0.0;
        for (int i = 0; i < s.N; ++i) {
            const double* v = &s.h_vel[(size_t)i * 3];
            t += (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * 1.0;
        }
        if (!(cm.allreduce_sum(ng, 2) && cm.allreduce_sum(&t, 1))) {
            set_error(MD_ERR_COMM, "md_report_particles: " + cm.error());
            return;
        }
        if (cm.rank() != 0) return;
        std::printf("# Local # Ghost Temp\n");
        std::printf("%lld %lld ", ng[0], ng[1]);
        print_g(t * (1.0 / (double)(ng[0] * 3 - 3)));
        std::printf("\n");
        std::fflush(stdout);
        return;
    }
    std::printf("# Local # Ghost Temp\n");
    std::printf("%d %d ", s.N, s.G);
    print_g(host_temperature(s));
    std::printf("\n");
    std::fflush(stdout);
}

// core/runtime.impala:318-337
void md_report_time(double total, double force, double neigh, double comm_t, double lb, double other) {
    double v[6] = {total, force, neigh, comm_t, lb, other};
    Comm& cm = comm();  // the slowest rank's times, printed once
    if (cm.active() && !cm.allreduce_max(v, 6)) set_error(MD_ERR_COMM, "md_report_time: " + cm.error());
    if (cm.rank() != 0) return;
    std::printf("Total Force Neigh Comm Balance Other\n");
    for (double x : v) {
        print_g(x);
        std::printf(" ");
    }
    std::printf("\n");
    std::fflush(stdout);
}

// ---- extensions ---------------------------------------------------------------
void md_set_precision(int mode) {
    State& s = g_state;
    mode = mode ? 1 : 0;
    if (s.alive && mode != s.precision) {
        flush_all(s);
        const int NA = s.N + s.G;
        if (NA > 0) {
            launch(s, (NA + 255) / 256, 256, 0, k_convert_forces, s.frc.b[s.ac], s.frc32, NA, mode);
            launched(K_MISC);
        }
        s.precision = mode;
        if (mode == 1) run_refresh_pos32(s);
    }
    s.precision = mode;
}
void md_set_half_mode(int ghost_pairs) {
    if (g_state.alive) flush_all(g_state);
    g_state.half_ghost = ghost_pairs ? 1 : 0;
    g_state.lists_valid = 0;
}
void md_set_ghost_mode(int exact) {
    if (g_state.alive) flush_all(g_state);
    g_state.ghost_exact = (exact || g_state.halo.on) ? 1 : 0;  // several ranks: exact ghosts only
}
void md_set_dem_model(int fixed, double radius) {
    if (g_state.alive) flush_all(g_state);
    g_state.dem_fixed = fixed ? 1 : 0;
    g_state.dem_radius = radius;
}
void md_set_thermo(int enable) {
    if (g_state.alive) flush_all(g_state);
    g_state.thermo = enable ? 1 : 0;
}
int md_get_thermo(double* out) {
    State& s = g_state;
    if (!require_alive("md_get_thermo")) return -1;
    flush_all(s);
    flush_thermo(s);
    TMD_CUDA(cudaMemcpyAsync(out, s.thermo_dev, 4 * sizeof(double), cudaMemcpyDeviceToHost, s.stream));
    sync_stream(s);
    s.rsq_iters = (long long)out[2];
    if (comm().active() && !comm().allreduce_sum(out, 4)) {  // every rank's sums
        set_error(MD_ERR_COMM, "md_get_thermo: " + comm().error());
        return -1;
    }
    return 0;
}
// Asynchronous thermo: the sums as of the work enqueued so far go to a page-locked slot by a
// copy on the library stream, gated by an event; nothing waits until the ticket is fetched.
int md_thermo_request(void) {
    State& s = g_state;
    if (!require_alive("md_thermo_request")) return -1;
    flush_all(s);
    flush_thermo(s);
    const long long t = s.thermo_tickets++;
    const int k = (int)(t % kThermoSlots);
    if (s.thermo_slot_ticket[k] >= 0) TMD_CUDA(cudaEventSynchronize(s.thermo_ev[k]));  // slot reused
    TMD_CUDA(cudaMemcpyAsync(s.thermo_host + 4 * k, s.thermo_dev, 4 * sizeof(double), cudaMemcpyDeviceToHost,
                             s.stream));
    TMD_CUDA(cudaEventRecord(s.thermo_ev[k], s.stream));
    s.thermo_slot_ticket[k] = t;
    return (int)t;
}
int md_thermo_fetch(int ticket, double* out) {
    State& s = g_state;
    if (!require_alive("md_thermo_fetch")) return -1;
    const int k = ticket >= 0 ? ticket % kThermoSlots : 0;
    if (ticket < 0 || s.thermo_slot_ticket[k] != ticket) {
        set_error(MD_ERR_ARGUMENT, "md_thermo_fetch: unknown ticket (more than 8 requests since, or none)");
        return -1;
    }
    TMD_CUDA(cudaEventSynchronize(s.thermo_ev[k]));
    for (int q = 0; q < 4; ++q) out[q] = s.thermo_host[4 * k + q];
    s.rsq_iters = (long long)out[2];
    if (comm().active() && !comm().allreduce_sum(out, 4)) {  // every rank fetches the same tickets
        set_error(MD_ERR_COMM, "md_thermo_fetch: " + comm().error());
        return -1;
    }
    return 0;
}
void md_synchronize(void) {
    if (g_state.alive) {
        flush_all(g_state);
        sync_stream(g_state);
    }
}
void md_get_phase_times(double* out) {
    if (g_state.alive) flush_all(g_state);
    phase_times(out);
}
void md_profile_enable(int mask) {
    if (g_state.alive) flush_all(g_state);
    prof_mask = mask;
}
void md_set_phase_timing(int enable) {
    if (g_state.alive) flush_all(g_state);
    phase_on = enable != 0;
    if (!phase_on) cur_phase = 0;
}
void md_profile_sample(int every) {
    if (g_state.alive) flush_all(g_state);
    prof_every = every > 0 ? every : 1;
}
int md_profile_count(void) { return K_COUNT; }
const char* md_profile_name(int id) { return kernel_name(id); }
int md_profile_get(int id, long long* launches, double* total_ms) {
    if (id < 0 || id >= K_COUNT) return -1;
    if (g_state.alive) flush_all(g_state);
    fold_prof(true);
    *launches = prof_launch[id];
    *total_ms = prof_ms[id];
    return 0;
}
void md_profile_reset(void) { prof_reset(); }
long long md_kernel_launches(void) { return g_state.launches; }
long long md_device_bytes(void) { return g_state.dev_bytes; }
void md_release_device_memory(void) { release_kept_blocks(); }

int md_get_neighbor_lists(int* sizes, int* lists, int capacity) {
    State& s = g_state;
    if (!require_alive("md_get_neighbor_lists")) return -1;
    flush_all(s);
    one_sided_lists(s);
    const int N = s.N, NA = s.N + s.G;
    std::vector<int> n(N), ref(NA);
    std::vector<uint32_t> l((size_t)s.nb_cap * s.nb_stride);
    TMD_CUDA(cudaMemcpyAsync(n.data(), s.nbn, sizeof(int) * N, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(ref.data(), s.ref.b[s.ac], sizeof(int) * NA, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(l.data(), s.nbl, sizeof(uint32_t) * l.size(), cudaMemcpyDeviceToHost, s.stream));
    sync_stream(s);
    int mx = 0;
    for (int slot = 0; slot < N; ++slot) {
        const int r = ref[slot];
        sizes[r] = n[slot];
        mx = std::max(mx, n[slot]);
        for (int k = 0; k < n[slot] && k < capacity && k < s.nb_cap; ++k)
            lists[(size_t)r * capacity + k] = ref[l[(((size_t)(k >> 2) * s.nb_stride + slot) << 2) + (k & 3)] >> kCodeBits];
    }
    return mx;
}

int md_get_ghost_info(int* src, int* pbc, int* root, int* tshift) {
    State& s = g_state;
    if (!require_alive("md_get_ghost_info")) return -1;
    flush_all(s);
    const int G = s.G;
    std::vector<int> a(G), b(G), c(G);
    if (G) {
        TMD_CUDA(cudaMemcpyAsync(a.data(), s.bsrc_ref, sizeof(int) * G, cudaMemcpyDeviceToHost, s.stream));
        TMD_CUDA(cudaMemcpyAsync(b.data(), s.broot_ref, sizeof(int) * G, cudaMemcpyDeviceToHost, s.stream));
        TMD_CUDA(cudaMemcpyAsync(c.data(), s.bcode, sizeof(int) * G, cudaMemcpyDeviceToHost, s.stream));
        sync_stream(s);
    }
    for (int g = 0; g < G; ++g) {
        src[g] = a[g];
        root[g] = b[g];
        for (int d = 0; d < 3; ++d) {
            pbc[3 * g + d] = ((c[g] >> (2 * d)) & 3) - 1;
            tshift[3 * g + d] = ((c[g] >> (8 + 2 * d)) & 3) - 1;
        }
    }
    return G;
}

int md_get_state(double* pos, double* vel, double* frc) {
    State& s = g_state;
    if (!require_alive("md_get_state")) return -1;
    Snapshot sn;
    snapshot(s, sn);
    for (int slot = 0; slot < s.N + s.G; ++slot) {
        const int r = sn.ref[slot];
        if (pos) {
            pos[3 * r] = sn.pos[slot].x;
            pos[3 * r + 1] = sn.pos[slot].y;
            pos[3 * r + 2] = sn.pos[slot].z;
        }
        if (r >= s.N) continue;
        if (vel) {
            vel[3 * r] = sn.vel[slot].x;
            vel[3 * r + 1] = sn.vel[slot].y;
            vel[3 * r + 2] = sn.vel[slot].z;
        }
        if (frc) {
            if (s.precision == 1) {
                frc[3 * r] = sn.frc32[slot].x;
                frc[3 * r + 1] = sn.frc32[slot].y;
                frc[3 * r + 2] = sn.frc32[slot].z;
            } else {
                frc[3 * r] = sn.frc[slot].x;
                frc[3 * r + 1] = sn.frc[slot].y;
                frc[3 * r + 2] = sn.frc[slot].z;
            }
        }
    }
    return s.N + s.G;
}

static int set_local_vec(const double* in, bool is_pos) {
    State& s = g_state;
    if (!require_alive("md_set_positions")) return -1;
    flush_all(s);
    const int N = s.N;
    std::vector<int> sor(N);
    std::vector<double4> buf(N);
    double4* dst = is_pos ? s.pos.b[s.pc] : s.vel.b[s.vc];
    TMD_CUDA(cudaMemcpyAsync(sor.data(), s.slot_of_ref, sizeof(int) * N, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(buf.data(), dst, sizeof(double4) * N, cudaMemcpyDeviceToHost, s.stream));
    sync_stream(s);
    for (int r = 0; r < N; ++r) {
        double4& q = buf[sor[r]];
        q.x = in[3 * r];
        q.y = in[3 * r + 1];
        q.z = in[3 * r + 2];
    }
    TMD_CUDA(cudaMemcpyAsync(dst, buf.data(), sizeof(double4) * N, cudaMemcpyHostToDevice, s.stream));
    sync_stream(s);
    if (is_pos && s.precision == 1) run_refresh_pos32(s);
    return 0;
}
int md_set_positions(double const* pos) { return set_local_vec(pos, true); }
int md_set_velocities(double const* vel) { return set_local_vec(vel, false); }

int md_get_cell_sizes(int* out, int ncells) {
    State& s = g_state;
    if (!require_alive("md_get_cell_sizes")) return -1;
    flush_all(s);
    const int nc = s.geo.ncells;
    std::vector<int> c(2 * (nc + 1));
    TMD_CUDA(cudaMemcpyAsync(c.data(), s.cnt, sizeof(int) * c.size(), cudaMemcpyDeviceToHost, s.stream));
    sync_stream(s);
    for (int k = 0; k < nc && k < ncells; ++k) out[k] = c[k] + c[nc + 1 + k];
    return nc;
}

// Reads a buffer (L2 flush for benchmarking, after it was written): the written lines are
// evicted and written back here, outside any timed interval, and the cache is left holding
// clean lines of the buffer.  The sum only keeps the loads alive.
__global__ void k_l2_read(const uint4* __restrict__ b, size_t n, unsigned* __restrict__ sink) {
    unsigned acc = 0;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const uint4 v = __ldcg(b + k);
        acc ^= v.x ^ v.y ^ v.z ^ v.w;
    }
    if (acc == 0x9e3779b9u) atomicAdd(sink, 1u);  // practically never: a side effect the compiler keeps
}

// The md driver's timestep loop (main.cpp:715-776) issued natively.
int md_run_timesteps(int steps, double dt, int reneigh_every, int step0, double list_cutoff, float* step_ms,
                     void* flush_buf, long long flush_bytes) {
    Range range("md_run_timesteps");
    State& s = g_state;
    if (!require_alive("md_run_timesteps")) return -1;
    if (!s.force_cfg.valid || reneigh_every <= 0 || steps < 0) {
        set_error(MD_ERR_STATE, "md_run_timesteps: no force configured (call md_compute_* once) or bad arguments");
        return -1;
    }
    flush_all(s);
    std::vector<cudaEvent_t> ev;
    if (step_ms) {
        ev.resize(2 * (size_t)steps);
        for (auto& e : ev) TMD_CUDA(cudaEventCreate(&e));
    }
    const PendingForce cfg = s.force_cfg;
    for (int k = 0; k < steps; ++k) {
        if (flush_buf && flush_bytes > 0) {
            TMD_CUDA(cudaMemsetAsync(flush_buf, (k & 0x7f) + 1, (size_t)flush_bytes, s.stream));
            k_l2_read<<<148 * 8, 256, 0, s.stream>>>(static_cast<const uint4*>(flush_buf), (size_t)flush_bytes / 16,
                                                     reinterpret_cast<unsigned*>(s.thermo_dev + 7));
        }
        if (step_ms) TMD_CUDA(cudaEventRecord(ev[2 * k], s.stream));
        md_initial_integration(dt);
        if ((step0 + k + 1) % reneigh_every == 0) {
            md_exchange_particles();
            md_enforce_pbc();
            md_borders();
            md_distribute_particles();
            md_assemble_neighborlists(cfg.half, list_cutoff);
        } else {
            md_synchronize_ghost_layer();
        }
        if (cfg.dem) md_compute_dem(cfg.half, cfg.rc, cfg.dn, cfg.dt_, cfg.k, cfg.mu);
        else md_compute_lennard_jones(cfg.half, cfg.rc, cfg.eps, cfg.sigma);
        md_final_integration(dt);
        if (k == steps - 1) flush_all(s);  // the last step's force is inside its time
        if (step_ms) TMD_CUDA(cudaEventRecord(ev[2 * k + 1], s.stream));
    }
    sync_stream(s);
    for (int k = 0; step_ms && k < steps; ++k) {
        float ms = 0.f;
        TMD_CUDA(cudaEventElapsedTime(&ms, ev[2 * k], ev[2 * k + 1]));
        step_ms[k] = ms;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    return s.last_error == MD_ERR_CUDA ? -1 : 0;
}

// several ranks: this rank's own periodic ghosts, images sent and ghosts received per step,
// neighbour ranks (the halo's size: (sent + received) x 24 bytes per step)
int tmd_halo_info(int* out) {
    const Halo& h = g_state.halo;
    out[0] = h.gself;
    out[1] = h.nsend;
    out[2] = h.nrecv;
    out[3] = (int)comm().topo.peers.size();
    return h.on ? 0 : -1;
}

int md_get_grid_info(int* out) {
    State& s = g_state;
    out[0] = s.geo.nx;
    out[1] = s.geo.ny;
    out[2] = s.geo.nz;
    out[3] = s.geo.ncells;
    out[4] = s.N;
    out[5] = s.G;
    out[6] = s.nb_cap;
    out[7] = s.nb_stride;
    return 0;
}

}  // extern "C"
