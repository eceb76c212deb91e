// adjoint.cu -- the differentiable form: gradients of a trajectory loss with
// respect to the initial velocities, epsilon and sigma by reverse-mode
// differentiation of velocity-Verlet with LJ over full neighbour lists.
//
// Trajectory (the md driver loop, main.cpp:715-776, with exact periodic
// ghosts): v_h = v_t + c F(x_t); x_{t+1} = x_t + dt v_h; v_{t+1} = v_h + c F(x_{t+1}),
// c = dt/2, lists rebuilt (after a periodic wrap) whenever (t+1) % R == 0.
// Loss: L = (1/N) sum_i |x_T,i - x_0,i|^2 (unwrapped) + U(x_T)/N.
//
// Reverse pass.  With a_x = dL/dx_t and a_v = dL/dv_t, one step back is
//   a_x += c J(x_{t+1}) a_v ; a_v += dt a_x ; a_x += c J(x_t) a_v ; (theta: c dF/dtheta^T a_v at both)
// where J = dF/dx = -Hessian.  The product J(x_t) a_v(t) appears in step t
// (initial kick) and step t-1 (final kick), so one Hessian-vector product per
// step suffices: k_adj_hvp_split computes u = J(x_t) a_v, adds dt*u (c*u at t = 0)
// to a_x, applies the next drift a_v += dt a_x, and accumulates the theta
// terms with weight dt (c at t = 0) into per-block sums (deterministic).
//
// Memory: a checkpoint (positions, velocities, wrap counts in reference
// order) per reneighbour segment; the backward pass restores a segment,
// rebuilds its cells / ghosts / list (bit-identical to the forward's: all are
// keyed by reference index) and recomputes the segment's positions with the
// same kernels, so the recomputed trajectory is the forward one bit for bit.

#include <cmath>
#include <cstdio>
#include <utility>
#include <vector>

#include "md_common.cuh"
#include "comm.h"
#include "launch.cuh"
#include "md_state.h"
#include "tinymd_b200.h"

namespace tmd {

bool grow_atoms(State& s, int need);

namespace {

constexpr int kT = 256;

struct AdjConfig {
    bool configured = false;
    int steps = 0, reneigh = 20, precision = 1;
    int shifted = 0;  // loss energy shifted to zero at the cutoff (continuous)
    double dt = 0.005, cutoff = 2.5, skin = 0.3;
};

struct AdjRun {
    bool forward_done = false;
    double eps = 1.0, sigma = 1.0, loss = 0.0, U = 0.0;
    int nseg = 0;
    double fwd_ms = 0.0, bwd_ms = 0.0;
};

AdjConfig cfg;
AdjRun run;

// device buffers (sized N or N+G)
double4* ck_x = nullptr;   // [nseg][N] positions, reference order
double4* ck_v = nullptr;   // [nseg][N] velocities
int* ck_img = nullptr;     // [nseg][N] wrap counts
double4* x0_dev = nullptr; // [N] initial positions, reference order
double4* seg_x = nullptr;  // [reneigh][N + G] positions (ghosts too) of one segment, slot order
int* nbr = nullptr;        // root slot of each list entry, laid out as the list
size_t cap_nbr = 0;
double4* ax = nullptr;     // [N] adjoint of positions, slot order
double4* av[2] = {nullptr, nullptr};
double4* tmp4 = nullptr;   // [N] reference-order staging
double* gacc = nullptr;    // [3][nblk] per-block theta sums (eps, sigma, unused)
double* red = nullptr;     // [8] reduced sums
int cap_n = 0, cap_seg = 0, cap_ck = 0;

inline int nblk(long long n) { return (int)((n + kT - 1) / kT); }

// Lanes per atom of the product kernel: more lanes shorten the chain of gathers and FP64 pair terms
// that bounds a small system.  Kernel times in us by CUDA events (5 us of them the events), 4 / 8 / 16 /
// 32 lanes: 864 atoms 16.7 / 12.7 / 10.8 / 9.0, 4,000 17.1 / 12.9 / 11.3 / 14.8, 8,788 17.0 / 14.5 / 16.9,
// 16,384 19.0 / 21.1 / 23.1, 70,304 47.5 / 51.2 / 66.6.
inline int hvp_lanes(int N) { return N <= 3000 ? 32 : N <= 6000 ? 16 : N <= 12000 ? 8 : 4; }

struct HvpArgs {
    int N, stride, nbcap;
    double rc2, sigma6, eps, inv_sigma;
    double len[3];
    double kick;       // added to a_x: dt * u (c * u at t = 0)
    double drift;      // a_v += drift * a_x after the kick (0 at t = 0)
    double wt;         // weight of this position's theta terms
};

// u_i = sum_j [f(s) w_ij + 2 f'(s) (d . w_ij) d],  w_ij = w_i - w_j, d = x_i - x_j,
// f = 48 eps sr6 (sr6 - 1/2) sr2, f' = df/ds = 48 eps sr2^2 sr6 (2 - 7 sr6);
// theta terms: sum_j f (d . w_i) / eps (= w_i . F_i / eps) and sum_j df/dsigma (d . w_i),
// df/dsigma = (144 eps / sigma) sr2 sr6 (4 sr6 - 1).
// The neighbour loop is split over kLpa adjacent lanes per atom (hvp_lanes; lane
// `sub` takes entries sub, sub + kLpa, ...) in batches of kHb with the next batch's
// entries loaded ahead, and the lanes' sums combined by shuffles.  Ghost neighbours
// read their stored position (xs holds all slots of the step) and the adjoint of
// their root through the root list `nbr`, so a neighbour costs two independent gathers.
constexpr int kHb = 2;  // neighbours per lane per batch (3 and 4: 110 registers, 47.5 -> 53.8 us at 70,304 atoms)

template <int kLpa>
__global__ void __launch_bounds__(kT)
k_adj_hvp_split(const double4* __restrict__ xs, const double4* __restrict__ w, double4* __restrict__ w_next,
                double4* __restrict__ ax, const int* __restrict__ nbn, const uint32_t* __restrict__ nbl,
                const int* __restrict__ nbr, double* __restrict__ gacc, HvpArgs a) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ double scratch[kT / 32];
    const int t = blk * blockDim.x + threadIdx.x;
    const int i = t / kLpa, sub = t % kLpa;
    const bool act = i < a.N;
    double ux = 0.0, uy = 0.0, uz = 0.0, ge = 0.0, gs = 0.0;
    double4 wi = make_double4(0.0, 0.0, 0.0, 0.0);
    if (act) {
        const double4 xi = ldg_d4(xs + i);
        wi = ldg_d4(w + i);
        const int n = min(nbn[i], a.nbcap);
        int ej[kHb], er[kHb];
#pragma unroll
        for (int b = 0; b < kHb; ++b) {
            const int k = sub + b * kLpa;
            ej[b] = k < n ? (int)(__ldg(nbl + nl_index(k, i, a.stride)) >> kCodeBits) : i;
            er[b] = k < n ? __ldg(nbr + nl_index(k, i, a.stride)) : i;
        }
        for (int k0 = sub; k0 < n; k0 += kLpa * kHb) {
            double4 xj[kHb], wj[kHb];
#pragma unroll
            for (int b = 0; b < kHb; ++b) {
                xj[b] = ldg_d4(xs + ej[b]);
                wj[b] = ldg_d4(w + er[b]);
            }
#pragma unroll
            for (int b = 0; b < kHb; ++b) {
                const int k = k0 + kLpa * kHb + b * kLpa;
                ej[b] = k < n ? (int)(__ldg(nbl + nl_index(k, i, a.stride)) >> kCodeBits) : i;
                er[b] = k < n ? __ldg(nbr + nl_index(k, i, a.stride)) : i;
            }
#pragma unroll
            for (int b = 0; b < kHb; ++b) {
                if (k0 + b * kLpa >= n) continue;
                const double dx = xi.x - xj[b].x, dy = xi.y - xj[b].y, dz = xi.z - xj[b].z;
                const double s = dx * dx + dy * dy + dz * dz;
                if (s < a.rc2) {
                    const double sr2 = 1.0 / s;
                    const double sr6 = sr2 * sr2 * sr2 * a.sigma6;
                    const double f = 48.0 * a.eps * sr6 * (sr6 - 0.5) * sr2;
                    const double fp = 48.0 * a.eps * sr2 * sr2 * sr6 * (2.0 - 7.0 * sr6);
                    const double wx = wi.x - wj[b].x, wy = wi.y - wj[b].y, wz = wi.z - wj[b].z;
                    const double dw = 2.0 * fp * (dx * wx + dy * wy + dz * wz);
                    const double di = dx * wi.x + dy * wi.y + dz * wi.z;
                    ux += f * wx + dw * dx;
                    uy += f * wy + dw * dy;
                    uz += f * wz + dw * dz;
                    ge += f * di;
                    gs += 144.0 * a.eps * a.inv_sigma * sr2 * sr6 * (4.0 * sr6 - 1.0) * di;
                }
            }
        }
    }
#pragma unroll
    for (int o = 1; o < kLpa; o <<= 1) {
        ux += __shfl_xor_sync(0xffffffffu, ux, o);
        uy += __shfl_xor_sync(0xffffffffu, uy, o);
        uz += __shfl_xor_sync(0xffffffffu, uz, o);
    }
    ge /= a.eps;
    if (act && sub == 0) {
        double4 q = ld_d4(ax + i);
        q.x += a.kick * ux;
        q.y += a.kick * uy;
        q.z += a.kick * uz;
        st_d4(ax + i, q);
        st_d4(w_next + i, make_double4(wi.x + a.drift * q.x, wi.y + a.drift * q.y, wi.z + a.drift * q.z, 0.0));
    }
    const double se = block_sum(ge, scratch);
    const double ss = block_sum(gs, scratch);
    if (threadIdx.x == 0) {
        gacc[blk] += a.wt * se;
        gacc[gridDim.x + blk] += a.wt * ss;
    }
}

// the root slot of every list entry (a ghost's root local, a local itself)
__global__ void k_root_list(const int* __restrict__ nbn, const uint32_t* __restrict__ nbl,
                            const int* __restrict__ groot, int* __restrict__ nbr, int N, int stride, int nbcap) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int i = blk * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int n = min(nbn[i], nbcap);
    for (int k = 0; k < n; ++k) {
        const int j = (int)(nbl[nl_index(k, i, stride)] >> kCodeBits);
        nbr[nl_index(k, i, stride)] = j < N ? j : groot[j - N];
    }
}

// loss pieces at x_T: MSD sum over locals, dU/dsigma sum, the pair energy (FP64, each
// pair seen from both atoms), and the initial adjoint a_x = (2/N)(x_T + img L - x_0) - F/N,
// a_v = dt a_x (drift of step T-1).  The three sums are compensated, per block as (sum,
// correction) rows of part: the loss enters central differences of ~1e-12.
__global__ void __launch_bounds__(kT)
k_adj_init(const double4* __restrict__ pos, const int* __restrict__ img, const int* __restrict__ ref,
           const double4* __restrict__ x0, const double4* __restrict__ frc, const float4* __restrict__ frc32,
           int mixed, const int* __restrict__ nbn, const uint32_t* __restrict__ nbl, double4* __restrict__ ax,
           double4* __restrict__ av, double* __restrict__ part, int N, int stride, int nbcap, double rc2,
           double sigma6, double eps, double inv_sigma, double len0, double len1, double len2, double dt) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ double scratch[64];
    const int i = blk * blockDim.x + threadIdx.x;
    double msd = 0.0, dus = 0.0, ue = 0.0, dus_c = 0.0, ue_c = 0.0, np_ = 0.0, np_c = 0.0;
    if (i < N) {
        const double4 p = pos[i];
        const int im = img[i];
        const double4 o = x0[ref[i]];
        const double ux = p.x + len0 * wrap_diff(unpack_axis(im, 0), 0) - o.x;
        const double uy = p.y + len1 * wrap_diff(unpack_axis(im, 1), 0) - o.y;
        const double uz = p.z + len2 * wrap_diff(unpack_axis(im, 2), 0) - o.z;
        msd = ux * ux + uy * uy + uz * uz;
        double fx, fy, fz;
        if (mixed) {
            fx = frc32[i].x; fy = frc32[i].y; fz = frc32[i].z;
        } else {
            fx = frc[i].x; fy = frc[i].y; fz = frc[i].z;
        }
        const double inv_n = 1.0 / N;
        const double4 a = make_double4(2.0 * inv_n * ux - fx * inv_n, 2.0 * inv_n * uy - fy * inv_n,
                                       2.0 * inv_n * uz - fz * inv_n, 0.0);
        ax[i] = a;
        av[i] = make_double4(dt * a.x, dt * a.y, dt * a.z, 0.0);
        const int n = min(nbn[i], nbcap);
        for (int k = 0; k < n; ++k) {
            const int j = (int)(__ldg(nbl + nl_index(k, i, stride)) >> kCodeBits);
            const double4 q = ldg_d4(pos + j);
            const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const double s = dx * dx + dy * dy + dz * dz;
            if (s < rc2) {
                const double sr2 = 1.0 / s;
                const double sr6 = sr2 * sr2 * sr2 * sigma6;
                // full list: 1/2 of 24 eps/sigma (...) and 1/2 of the pair energy
                dd_add(dus, dus_c, 12.0 * eps * inv_sigma * (2.0 * sr6 * sr6 - sr6), 0.0);
                dd_add(ue, ue_c, 2.0 * eps * sr6 * (sr6 - 1.0), 0.0);
                np_ += 0.5;  // pairs inside the cutoff (exact: halves of small integers)
            }
        }
    }
    double msd_c = 0.0;
    block_sum_dd(msd, msd_c, scratch);
    block_sum_dd(dus, dus_c, scratch);
    block_sum_dd(ue, ue_c, scratch);
    block_sum_dd(np_, np_c, scratch);
    if (threadIdx.x == 0) {
        const int nb = gridDim.x;
        part[blk] = msd;
        part[nb + blk] = msd_c;
        part[2 * nb + blk] = dus;
        part[3 * nb + blk] = dus_c;
        part[4 * nb + blk] = ue;
        part[5 * nb + blk] = ue_c;
        part[6 * nb + blk] = np_;
        part[7 * nb + blk] = np_c;
    }
}

// out[q] = the compensated total of rows (2q, 2q + 1) of part[.][nb]
__global__ void k_sum_rows_dd(const double* __restrict__ part, double* __restrict__ out, int nb, int nq) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ double scratch[64];
    for (int q = 0; q < nq; ++q) {
        double s = 0.0, c = 0.0;
        for (int b = threadIdx.x + blk; b < nb; b += blockDim.x) dd_add(s, c, part[2 * q * nb + b], part[(2 * q + 1) * nb + b]);
        block_sum_dd(s, c, scratch);
        if (threadIdx.x == 0) out[q] = s + c;
    }
}

__global__ void k_sum_rows(const double* __restrict__ part, double* __restrict__ out, int nb, int rows) {
    const int blk = (int)blockIdx.x + pdl_wait();
    __shared__ double scratch[32];
    for (int q = 0; q < rows; ++q) {
        double v = 0.0;
        for (int b = threadIdx.x + blk; b < nb; b += blockDim.x) v += part[q * nb + b];
        const double r = block_sum(v, scratch);
        if (threadIdx.x == 0) out[q] = r;
    }
}

// slot order -> reference order (locals)
__global__ void k_to_ref(const double4* __restrict__ src, const int* __restrict__ ref, double4* __restrict__ dst,
                         int N) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int s = blk * blockDim.x + threadIdx.x;
    if (s < N) st_d4(dst + ref[s], ldg_d4(src + s));
}
// reference order -> slot order (locals)
__global__ void k_from_ref(const double4* __restrict__ src, const int* __restrict__ ref, double4* __restrict__ dst,
                           int N) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int s = blk * blockDim.x + threadIdx.x;
    if (s < N) st_d4(dst + s, ldg_d4(src + ref[s]));
}
// checkpoint of the current state in reference order
__global__ void k_checkpoint(const double4* __restrict__ pos, const double4* __restrict__ vel,
                             const int* __restrict__ img, const int* __restrict__ ref, double4* __restrict__ cx,
                             double4* __restrict__ cv, int* __restrict__ ci, int N) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int s = blk * blockDim.x + threadIdx.x;
    if (s < N) {
        const int r = ref[s];
        st_d4(cx + r, ldg_d4(pos + s));
        st_d4(cv + r, ldg_d4(vel + s));
        ci[r] = img[s];
    }
}
// restore a checkpoint into the identity layout (slot = reference index)
__global__ void k_restore(const double4* __restrict__ cx, const double4* __restrict__ cv,
                          const int* __restrict__ ci, const double* __restrict__ mass_ref, double4* __restrict__ pos,
                          double4* __restrict__ vel, int* __restrict__ img, int* __restrict__ ref,
                          int* __restrict__ slot_of_ref, double* __restrict__ mass, int N) {
    const int blk = (int)blockIdx.x + pdl_wait();
    const int r = blk * blockDim.x + threadIdx.x;
    if (r < N) {
        st_d4(pos + r, ldg_d4(cx + r));
        st_d4(vel + r, ldg_d4(cv + r));
        img[r] = ci[r];
        ref[r] = r;
        slot_of_ref[r] = r;
        mass[r] = mass_ref[r];
    }
}

double* mass_ref = nullptr;

template <class T>
void ensure(T** p, int& cap, size_t need) {
    if ((size_t)cap >= need && *p) return;
    dfree(p);
    dalloc(p, need);
    cap = (int)need;
}

void free_adjoint() {
    dfree(&ck_x); dfree(&ck_v); dfree(&ck_img); dfree(&x0_dev); dfree(&seg_x); dfree(&nbr); dfree(&ax);
    dfree(&av[0]); dfree(&av[1]); dfree(&tmp4); dfree(&gacc); dfree(&red); dfree(&mass_ref);
    cap_n = cap_seg = cap_ck = 0;
    cap_nbr = 0;
}

// the list and layout for positions at the start of a segment (already wrapped)
void rebuild(State& s) {
    run_borders(s);
    run_distribute(s);
    run_build_lists(s, false, cfg.cutoff + cfg.skin);
}

void reset_identity(State& s, int ckpt) {
    const int N = s.N;
    s.G = 0;
    s.pc = s.vc = s.ac = 0;
    launch(s, nblk(N), kT, 0, k_restore, ck_x + (size_t)ckpt * N, ck_v + (size_t)ckpt * N, ck_img + (size_t)ckpt * N,
           mass_ref, s.pos.b[0], s.vel.b[0], s.img.b[0], s.ref.b[0], s.slot_of_ref, s.mass.b[0], N);
    launched(K_ADJ_STEP);
}

PendingForce force_params() {
    PendingForce p;
    p.valid = true;
    p.rc = cfg.cutoff;
    p.eps = run.eps;
    p.sigma = run.sigma;
    return p;
}

void checkpoint(State& s, int k) {
    const int N = s.N;
    launch(s, nblk(N), kT, 0, k_checkpoint, s.pos.b[s.pc], s.vel.b[s.vc], s.img.b[s.ac], s.ref.b[s.ac],
           ck_x + (size_t)k * N, ck_v + (size_t)k * N, ck_img + (size_t)k * N, N);
    launched(K_ADJ_STEP);
}

// the ghosts and lists after an integration to x_{t+1}: rebuilt when (t+1) % R == 0, else the ghosts
// refreshed where the integrating kernel has not written them
void finish_move(State& s, int t, bool pushed) {
    if ((t + 1) % cfg.reneigh == 0) {
        run_enforce_pbc(s);
        rebuild(s);
    } else if (!pushed && s.ghosts_pushed != 2) {
        run_ghost_refresh(s, 2);
    }
}

// The velocity-Verlet steps t0 .. t1-1 from x_t0 (with its force) on: one kernel per step, the force at
// x_{t+1}, its kick and the integration to x_{t+2}, as the driver's loop runs it; after_step(t) is called
// with x_{t+1}, v_{t+1} in place wherever stop(t) asks for it, and after the last step.  move(t) is
// called before the launch that writes x_{t+1}.  With the contact model set the force and the integration
// run apart: only run_integrate refreshes the ghosts' velocities, which that model's grid holds.
template <class Stop, class After, class Move>
void run_steps(State& s, int t0, int t1, bool last_force, Stop stop, After after_step, Move move) {
    bool moved = false;  // x_{t+1} is there already
    for (int t = t0; t < t1; ++t) {
        if (!moved) {
            move(t);
            const bool ren = (t + 1) % cfg.reneigh == 0;
            run_integrate(s, cfg.dt, !ren);
            finish_move(s, t, true);
        }
        moved = t + 1 < t1 && !stop(t) && s.dem_fixed == 0;
        if (moved) {
            move(t + 1);
            run_force_lj_init(s, force_params(), cfg.dt, cfg.dt);
            finish_move(s, t + 1, false);
        } else if (t + 1 < t1 || last_force) {
            run_force_lj(s, force_params(), true, cfg.dt);
            after_step(t);
        }
    }
}

struct ModeGuard {  // the adjoint runs exact ghosts, full lists, its own precision, no thermo
    int prec, ghost, thermo, half;
    explicit ModeGuard(State& s) : prec(s.precision), ghost(s.ghost_exact), thermo(s.thermo), half(s.half_ghost) {
        s.precision = cfg.precision;
        s.ghost_exact = 1;
        s.thermo = 0;
        s.half_ghost = 0;
    }
    void restore(State& s) {
        s.precision = prec;
        s.ghost_exact = ghost;
        s.thermo = thermo;
        s.half_ghost = half;
    }
};

}  // namespace

// the adjoint's device buffers (checkpoints, adjoints, root lists) go with the grid
void release_adjoint() { free_adjoint(); }

}  // namespace tmd

using namespace tmd;

extern "C" {

int md_adjoint_configure(int steps, int reneigh, double dt, double cutoff, double skin, int precision) {
    if (comm().active()) {  // the trajectory is one rank's periodic box
        set_error(MD_ERR_UNSUPPORTED, "md_adjoint_configure: the differentiable form runs on one rank");
        return -1;
    }
    if (steps < 1 || reneigh < 1 || !(dt > 0) || !(cutoff > 0) || skin < 0) {
        set_error(MD_ERR_ARGUMENT, "md_adjoint_configure: invalid arguments");
        return -1;
    }
    cfg.configured = true;
    cfg.steps = steps;
    cfg.reneigh = reneigh;
    cfg.dt = dt;
    cfg.cutoff = cutoff;
    cfg.skin = skin;
    cfg.precision = precision ? 1 : 0;
    run.forward_done = false;
    return 0;
}

int md_adjoint_forward(double const* v0, double epsilon, double sigma, double* loss) {
    State& s = g_state;
    if (!s.alive || !cfg.configured) {
        set_error(MD_ERR_STATE, "md_adjoint_forward: initialise the grid and call md_adjoint_configure first");
        return -1;
    }
    md_synchronize();
    const int N = s.N;
    run.eps = epsilon;
    run.sigma = sigma;
    run.nseg = (cfg.steps + cfg.reneigh - 1) / cfg.reneigh;
    ensure(&ck_x, cap_ck, (size_t)run.nseg * N);
    dfree(&ck_v);
    dfree(&ck_img);
    dalloc(&ck_v, (size_t)run.nseg * N);
    dalloc(&ck_img, (size_t)run.nseg * N);
    dfree(&x0_dev);
    dalloc(&x0_dev, N);
    dfree(&mass_ref);
    dalloc(&mass_ref, N);
    // the reverse pass's buffers too, so that nothing waits for the device behind the steps
    const int nbs = nblk((long long)hvp_lanes(N) * N);  // blocks of its product kernel
    for (double4** p : {&ax, &av[0], &av[1], &tmp4}) {
        dfree(p);
        dalloc(p, N);
    }
    dfree(&gacc);
    dalloc(&gacc, 2 * (size_t)nbs + 2);
    dfree(&red);
    dalloc(&red, 8);
    // initial state in reference order: x_0 from md_initialize_grid, v_0 from the caller
    materialize_mirror(s);
    const double* x0 = s.x0_in_pos ? s.h_pos.data() : s.h_x0.data();
    std::vector<double4> hx(N), hv(N);
    for (int i = 0; i < N; ++i) {
        hx[i] = make_double4(x0[3 * i], x0[3 * i + 1], x0[3 * i + 2], 0.0);
        hv[i] = make_double4(v0[3 * i], v0[3 * i + 1], v0[3 * i + 2], 0.0);
    }
    std::vector<double> hm(s.h_mass.begin(), s.h_mass.begin() + N);
    TMD_CUDA(cudaMemcpyAsync(x0_dev, hx.data(), sizeof(double4) * N, cudaMemcpyHostToDevice, s.stream));
    TMD_CUDA(cudaMemcpyAsync(ck_x, hx.data(), sizeof(double4) * N, cudaMemcpyHostToDevice, s.stream));
    TMD_CUDA(cudaMemcpyAsync(ck_v, hv.data(), sizeof(double4) * N, cudaMemcpyHostToDevice, s.stream));
    TMD_CUDA(cudaMemsetAsync(ck_img, 0, sizeof(int) * N, s.stream));
    TMD_CUDA(cudaMemcpyAsync(mass_ref, hm.data(), sizeof(double) * N, cudaMemcpyHostToDevice, s.stream));
    ModeGuard guard(s);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s.stream);
    reset_identity(s, 0);
    rebuild(s);
    run_force_lj(s, force_params(), false, 0.0);
    auto checkpoint_after = [&](int t) { return (t + 1) % cfg.reneigh == 0 && t + 1 < cfg.steps; };
    run_steps(
        s, 0, cfg.steps, true, checkpoint_after,
        [&](int t) {
            if (checkpoint_after(t)) checkpoint(s, (t + 1) / cfg.reneigh);
        },
        [](int) {});
    cudaEventRecord(e1, s.stream);
    // loss: MSD and U at x_T, and the initial adjoint state
    const int nb = nblk(N);
    flush_thermo(s);  // sums of a forward run waiting in the scratch
    ensure_red_scratch(s, 8 * nb);
    const double sig6 = std::pow(sigma, 6);
    launch(s, nb, kT, 0, k_adj_init, s.pos.b[s.pc], s.img.b[s.ac], s.ref.b[s.ac], x0_dev, s.frc.b[s.ac], s.frc32,
           s.precision, s.nbn, s.nbl, ax, av[0], s.red_part, N, s.nb_stride, s.nb_cap, cfg.cutoff * cfg.cutoff, sig6,
           epsilon, 1.0 / sigma, s.geo.len[0], s.geo.len[1], s.geo.len[2], cfg.dt);
    launched(K_ADJ_STEP);
    launch(s, 1, 256, 0, k_sum_rows_dd, s.red_part, red, nb, 4);
    launched(K_ADJ_STEP);
    double sums[4] = {0, 0, 0, 0};
    TMD_CUDA(cudaMemcpyAsync(sums, red, sizeof(sums), cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaStreamSynchronize(s.stream));
    float fms = 0.f;
    cudaEventElapsedTime(&fms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    run.fwd_ms = fms;
    run.U = sums[2];  // FP64 pair energy of x_T (for both forward precisions), compensated
    double dUds = sums[1];
    if (cfg.shifted) {
        // U_s = U - (pairs inside the cutoff) * e_c, e_c = 4 eps ((sigma/rc)^12 - (sigma/rc)^6);
        const double pairs = sums[3];
        const double src6 = sig6 / std::pow(cfg.cutoff, 6);
        const double ec = 4.0 * epsilon * (src6 * src6 - src6);
        const double dec_ds = 4.0 * epsilon * (12.0 * src6 * src6 - 6.0 * src6) / sigma;
        run.U -= pairs * ec;
        dUds -= pairs * dec_ds;
    }
    run.loss = sums[0] / N + run.U / N;
    // the direct theta terms of U(x_T)/N; the reverse pass adds the trajectory terms
    std::vector<double> g0(2 * (size_t)nbs + 2, 0.0);
    g0[2 * (size_t)nbs] = run.U / (N * epsilon);
    g0[2 * (size_t)nbs + 1] = dUds / N;
    TMD_CUDA(cudaMemcpyAsync(gacc, g0.data(), sizeof(double) * g0.size(), cudaMemcpyHostToDevice, s.stream));
    // adjoint state to reference order (the backward pass starts in another layout)
    launch(s, nb, kT, 0, k_to_ref, ax, s.ref.b[s.ac], tmp4, N);
    launched(K_ADJ_STEP);
    std::swap(ax, tmp4);
    launch(s, nb, kT, 0, k_to_ref, av[0], s.ref.b[s.ac], tmp4, N);
    launched(K_ADJ_STEP);
    std::swap(av[0], tmp4);
    TMD_CUDA(cudaStreamSynchronize(s.stream));
    guard.restore(s);
    *loss = run.loss;
    run.forward_done = s.last_error != MD_ERR_CUDA;
    return run.forward_done ? 0 : -1;
}

int md_adjoint_backward(double* grad_v0, double* grad_eps, double* grad_sigma) {
    State& s = g_state;
    if (!run.forward_done) {
        set_error(MD_ERR_STATE, "md_adjoint_backward: run md_adjoint_forward first");
        return -1;
    }
    const int N = s.N;
    const int nb = nblk(N);
    const int lanes = hvp_lanes(N);
    const int nbs = nblk((long long)lanes * N);
    const int R = cfg.reneigh;
    ModeGuard guard(s);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s.stream);
    const double c = 0.5 * cfg.dt;
    int wcur = 0;  // av[wcur] holds a_v (reference order between segments)
    std::vector<const double4*> x_at;  // a segment's positions, step by step
    for (int seg = run.nseg - 1; seg >= 0; --seg) {
        const int t0 = seg * R;
        const int t1 = std::min(t0 + R, cfg.steps);  // positions x_t0 .. x_{t1-1}
        reset_identity(s, seg);
        rebuild(s);
        // this segment's slots (ghosts included) and its root list
        const int NA = N + s.G;
        if ((size_t)cap_seg < (size_t)R * NA || !seg_x) {
            dfree(&seg_x);
            cap_seg = R * (NA + NA / 8 + 256);
            dalloc(&seg_x, (size_t)cap_seg);
        }
        const size_t nl = (size_t)s.nb_cap * s.nb_stride;
        if (cap_nbr < nl || !nbr) {
            dfree(&nbr);
            dalloc(&nbr, nl);
            cap_nbr = nl;
        }
        launch(s, nb, kT, 0, k_root_list, s.nbn, s.nbl, s.groot, nbr, N, s.nb_stride, s.nb_cap);
        launched(K_ADJ_STEP);
        run_force_lj(s, force_params(), false, 0.0);
        // x_t0 stays in the position buffer; each later step writes its positions straight into its
        // own part of seg_x, which stands in for the buffer written
        double4* const own[2] = {s.pos.b[0], s.pos.b[1]};
        x_at.assign(1, s.pos.b[s.pc]);
        run_steps(
            s, t0, t1 - 1, seg == 0, [](int) { return false; }, [](int) {},
            [&](int t) {
                double4* next = seg_x + (size_t)(t + 1 - t0) * NA;
                s.pos.b[1 - s.pc] = next;
                x_at.push_back(next);
            });
        s.pos.b[0] = own[0];
        s.pos.b[1] = own[1];
        // adjoint state into this segment's slot order
        const int* ref = s.ref.b[s.ac];
        launch(s, nb, kT, 0, k_from_ref, ax, ref, tmp4, N);
        launched(K_ADJ_STEP);
        std::swap(ax, tmp4);
        launch(s, nb, kT, 0, k_from_ref, av[wcur], ref, tmp4, N);
        launched(K_ADJ_STEP);
        std::swap(av[wcur], tmp4);
        HvpArgs a;
        a.N = N;
        a.stride = s.nb_stride;
        a.nbcap = s.nb_cap;
        a.rc2 = cfg.cutoff * cfg.cutoff;
        a.sigma6 = std::pow(run.sigma, 6);
        a.eps = run.eps;
        a.inv_sigma = 1.0 / run.sigma;
        for (int d = 0; d < 3; ++d) a.len[d] = s.geo.len[d];
        for (int t = t1 - 1; t >= t0; --t) {
            a.kick = t > 0 ? cfg.dt : c;
            a.drift = t > 0 ? cfg.dt : 0.0;
            a.wt = t > 0 ? cfg.dt : c;
            prof_begin(K_HVP);
            auto product = [&](auto kernel) {
                launch(s, nbs, kT, 0, kernel, x_at[t - t0], av[wcur], av[1 - wcur], ax, s.nbn, s.nbl, nbr, gacc, a);
            };
            if (lanes == 32) product(k_adj_hvp_split<32>);
            else if (lanes == 16) product(k_adj_hvp_split<16>);
            else if (lanes == 8) product(k_adj_hvp_split<8>);
            else product(k_adj_hvp_split<4>);
            launched(K_HVP);
            prof_end(K_HVP);
            wcur = 1 - wcur;
        }
        if (seg == 0 && x_at.size() > 1)  // the grid is left at the last recomputed positions, in its own buffer
            TMD_CUDA(cudaMemcpyAsync(s.pos.b[s.pc], x_at.back(), sizeof(double4) * NA, cudaMemcpyDeviceToDevice,
                                     s.stream));
        launch(s, nb, kT, 0, k_to_ref, ax, ref, tmp4, N);
        launched(K_ADJ_STEP);
        std::swap(ax, tmp4);
        launch(s, nb, kT, 0, k_to_ref, av[wcur], ref, tmp4, N);
        launched(K_ADJ_STEP);
        std::swap(av[wcur], tmp4);
    }
    cudaEventRecord(e1, s.stream);
    // theta gradients: per-block sums plus the direct terms stored after them
    launch(s, 1, 256, 0, k_sum_rows, gacc, red, nbs, 2);
    launched(K_ADJ_STEP);
    double gsum[2] = {0, 0}, direct[2] = {0, 0};
    std::vector<double4> hv(N);
    TMD_CUDA(cudaMemcpyAsync(gsum, red, sizeof(gsum), cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(direct, gacc + 2 * (size_t)nbs, sizeof(direct), cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaMemcpyAsync(hv.data(), av[wcur], sizeof(double4) * N, cudaMemcpyDeviceToHost, s.stream));
    TMD_CUDA(cudaStreamSynchronize(s.stream));
    float bms = 0.f;
    cudaEventElapsedTime(&bms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    run.bwd_ms = bms;
    for (int i = 0; i < N; ++i) {
        grad_v0[3 * i] = hv[i].x;
        grad_v0[3 * i + 1] = hv[i].y;
        grad_v0[3 * i + 2] = hv[i].z;
    }
    *grad_eps = gsum[0] + direct[0];
    *grad_sigma = gsum[1] + direct[1];
    guard.restore(s);
    run.forward_done = false;  // the reverse pass consumed the adjoint state
    return s.last_error == MD_ERR_CUDA ? -1 : 0;
}

int md_adjoint_set_loss(int shifted_energy) {
    cfg.shifted = shifted_energy ? 1 : 0;
    run.forward_done = false;
    return 0;
}

int md_adjoint_times(double* forward_ms, double* backward_ms) {
    *forward_ms = run.fwd_ms;
    *backward_ms = run.bwd_ms;
    return 0;
}

}  // extern "C"
