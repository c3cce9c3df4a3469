// Differentiable run: forward steps that record a tape, and the hand-written
// reverse of each step (contact law, both half-kicks of nve/sphere, pressure,
// servo and remap x).  FP64 throughout; atoms in the caller's order; the
// contacts are a half pair list (i < j) sorted by (i, j), and every per-atom
// sum gathers over the pairs in a fixed order (pairs as i, then as j), so
// results are bit-reproducible and the reverse sees exactly the forward's
// values.
//
// Forward of step s (Simulation._sub_step_inner, simulation.py:205-247):
//   k_initial   (remap of step s - 1;) v += dtf f / m; x += dt v; w += dtf t / I;
//               displacement check                            (nve_sphere.py:56-80)
//   k_pairs     contacts on the tape's xh, vh, wh (hertz_history.py:92-157)
//   k_gather    f, t per atom; v += dtf f / m; w += dtf t / I; kinetic partials
//   k_servo     virial total, pressure, servo, new box        (deform_pressure.py:598-702)
//   k_remap     x from the old box into the new one           (deform_pressure.py:493-530),
//               once per queued run of steps: between them k_initial does it
// Reverse of step s: k_b_servo (with k_b_reduce's sums of step s + 1), k_b_final,
// k_b_pairs, k_b_atoms (gather, first half-kick, remap of step s - 1).
//
// What bounds these kernels: the FP64 pipe (one instruction of a warp every 16
// cycles per SM, 64 cycles to its result) and, below a few ten thousand
// spheres, the chain of such results.  Hence small blocks (two warps), so that
// a few thousand atoms already reach every SM; quotients and roots by the short
// forms of tmps_common.cuh; pairs out of contact dropped before the law, so that its warps run
// full; and few launches, queued by one call for a run of steps with no host
// synchronisation in between: a step whose displacement check fires marks the
// run and every later launch of it does nothing.
#include "tmps_adjoint.cuh"
#include "tmps_common.cuh"

using namespace tmps;
using namespace tmps_adj;

namespace {

constexpr int kBlk = 64;       // threads of the per-atom and per-pair kernels
constexpr int kPairTile = 128;  // pairs a block of the contact passes takes
constexpr int kSum = 256;       // atoms or pairs the forward's sums join first (see sum_groups)
constexpr int kOne = 512;      // threads of the one-block kernels
constexpr int kNG = 16;        // doubles per pair in the reverse's per-pair record

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

struct Work {
    double* fp;     // [3][P] pair force on a
    double* tp;     // [3][P] pair torque term (d x fs) / r
    double* gp;     // [16][P] per-pair adjoints for the gather
    double* partw;  // [6][2 groups of kSum pairs] pair virial partials
    double* partk;  // [6][4 groups of kSum atoms] kinetic partials; [6][nbA] remap partials
    double* partg;  // [8][nbP] parameter and image partials of the reverse
    double* wbar;   // [6] dL/d(virial total) of the current reverse step: at the base, where the calls of
                    // a linked run find it whatever their numbers of pairs
};

// Blocks of the forward's per-atom and per-pair passes: whole groups of kSum.
int blocks_a(int n) { return kSum / kBlk * grid_for(n, kSum); }
int blocks_p(int npairs) { return kSum / kPairTile * grid_for(npairs, kSum); }

Work carve(void* base, int n, int npairs) {
    const int nbA = blocks_a(n), nbP = blocks_p(npairs);
    char* p = static_cast<char*>(base);
    Work w;
    w.wbar = reinterpret_cast<double*>(p); p += align256(sizeof(double) * 8);
    w.fp = reinterpret_cast<double*>(p); p += align256(sizeof(double) * 3 * (size_t)npairs);
    w.tp = reinterpret_cast<double*>(p); p += align256(sizeof(double) * 3 * (size_t)npairs);
    w.gp = reinterpret_cast<double*>(p); p += align256(sizeof(double) * kNG * (size_t)npairs);
    w.partw = reinterpret_cast<double*>(p); p += align256(sizeof(double) * 6 * (size_t)nbP);
    w.partk = reinterpret_cast<double*>(p); p += align256(sizeof(double) * 6 * (size_t)nbA);
    w.partg = reinterpret_cast<double*>(p);
    return w;
}

size_t work_bytes(int n, int npairs) {
    const int nbA = blocks_a(n), nbP = blocks_p(npairs);
    return align256(sizeof(double) * 3 * (size_t)npairs) * 2 + align256(sizeof(double) * kNG * (size_t)npairs) +
           align256(sizeof(double) * 6 * (size_t)nbP) + align256(sizeof(double) * 6 * (size_t)nbA) +
           align256(sizeof(double) * 8 * (size_t)nbP) + align256(sizeof(double) * 8);
}

Params to_params(const tmps_adj_params& p) {
    Params q;
    q.kn = p.kn;
    q.kt = p.kt;
    q.gamman = p.gamman;
    q.gammat = p.gammat;
    q.xmu = p.xmu;
    q.dt = p.dt;
    q.limit_damping = p.limit_damping;
    q.ikt = 1.0 / p.kt;
    return q;
}

// Minimum image on a fully periodic orthogonal box (domain.py:389-500 with
// round(d / prd) taken as rint(d * (1 / prd)); they differ only within an ulp
// of half a box, which no listed pair is).
__device__ __forceinline__ void min_image(const double* prd, const double* iprd, double* d, double* nimg) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        nimg[c] = 0.0;  // below 0.49 of the period without asking
        if ((__double2hiint(d[c]) & 0x7fffffff) >= __double2hiint(0.49 * prd[c])) {
            nimg[c] = rint(d[c] * iprd[c]);
            d[c] -= nimg[c] * prd[c];
        }
    }
}

__device__ __forceinline__ double inertia(double m, double r) { return ((0.4 * m) * r) * r; }

// Sum over the blocks' partials [NV][nb] into out[NV]: one warp per component
// (warps first, first + 1, ...), eight loads of a lane in flight at once, four
// running sums and a shuffle tree (fixed order).
template <int NV>
__device__ void sum_partials(const double* part, int nb, double* out, int first) {
    const int c = (threadIdx.x >> 5) - first, lane = threadIdx.x & 31;
    if (c < 0 || c >= NV) return;
    const double* row = part + (size_t)c * nb;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k0 = lane; k0 < nb; k0 += 256) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = k0 + 32 * u < nb ? row[k0 + 32 * u] : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) s[u & 3] += v[u];
    }
    double t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) out[c] = t;
}

// The forward's virial: the servo feeds a pressure's last bits back into every
// position, and the radius adjoints of barely touching pairs show those, so the
// sums keep one order whatever the kernels' blocks are: a tree over each 32
// consecutive atoms or pairs, a tree over the eight of a group of kSum, the
// groups a lane stride apart one after another, a tree over the lanes.  A block
// of the passes takes those warps of a group that its tree joins first and
// writes their sum; PER consecutive sums here make a group (PER - 1 additions).
// One warp per component (warps first, first + 1, ...).
template <int PER>
__device__ void sum_groups(const double* part, int ng, double* out, int first) {
    const int c = (threadIdx.x >> 5) - first, lane = threadIdx.x & 31;
    if (c < 0 || c >= 6) return;
    const double2* row = reinterpret_cast<const double2*>(part + (size_t)c * PER * ng);
    double t = 0.0;
    for (int k0 = lane; k0 < ng; k0 += 128) {
        double2 v[4][PER / 2];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int h = 0; h < PER / 2; ++h)
                v[u][h] = k0 + 32 * u < ng ? row[(size_t)(k0 + 32 * u) * (PER / 2) + h] : make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            double g = v[u][0].x + v[u][0].y;
            if constexpr (PER == 4) g += v[u][1].x + v[u][1].y;
            t += g;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) out[c] = t;
}

// Programmatic dependent launch: wait for the kernel before to complete, then
// let the next one be scheduled.  Every kernel of this file does both in this
// order, so when a block starts, all but the kernel right before it have
// completed: what those wrote may be read, and worked on, before enter().  That
// holds within one call of the interface; the first launch of every call is
// made without the attribute (Chain), whatever the caller queued before it.  The
// launches of a step depend on one another in a chain, so for few spheres the
// time of a step is the sum of their load and FP64 latencies, and each kernel
// does here what does not need its predecessor.
__device__ __forceinline__ void enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A queued run of steps: `hit` is the step whose displacement check fired (0:
// none).  That step's later launches and every launch of a later step return.
struct Queue {
    int64_t hit, done;
};
__device__ __forceinline__ bool halted(const Queue* q) { return q && *(volatile const int64_t*)&q->hit != 0; }

// ------------------------------------------------------------------ pairs

__global__ void __launch_bounds__(128) k_pairs_build(int n, const double* __restrict__ x, const double* __restrict__ rad,
                                                     const tmps_adj_rec* __restrict__ box, double skin,
                                                     int32_t* __restrict__ count, const int32_t* __restrict__ ibeg,
                                                     int32_t* __restrict__ pi, int32_t* __restrict__ pj) {
    // All pairs by tiles of 128 candidates in shared memory; an FP32 screen
    // with a wide margin, then the exact FP64 test (neighbor.py:348-356).
    __shared__ float4 tile[128];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double prd[3], iprd[3];
    float prd32[3], iprd32[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        prd[c] = box->prd[c];
        iprd[c] = 1.0 / prd[c];
        prd32[c] = (float)prd[c];
        iprd32[c] = (float)iprd[c];
    }
    const bool act = i < n;
    double xi[3] = {0, 0, 0}, ri = 0.0;
    if (act) {
        xi[0] = x[i];
        xi[1] = x[n + i];
        xi[2] = x[2 * n + i];
        ri = rad[i];
    }
    const float xi32[3] = {(float)xi[0], (float)xi[1], (float)xi[2]};
    int cnt = 0;
    int out = (act && pj) ? ibeg[i] : 0;
    const int j0 = blockIdx.x * blockDim.x;  // no candidate below the block's first atom can be above i
    for (int base = j0; base < n; base += 128) {
        __syncthreads();
        const int jl = base + threadIdx.x;
        if (jl < n) tile[threadIdx.x] = make_float4((float)x[jl], (float)x[n + jl], (float)x[2 * n + jl], (float)rad[jl]);
        __syncthreads();
        if (!act) continue;
        const int m = min(128, n - base);
        for (int k = 0; k < m; ++k) {
            const int j = base + k;
            if (j <= i) continue;
            const float4 q = tile[k];
            float d0 = xi32[0] - q.x, d1 = xi32[1] - q.y, d2 = xi32[2] - q.z;
            d0 -= prd32[0] * rintf(d0 * iprd32[0]);
            d1 -= prd32[1] * rintf(d1 * iprd32[1]);
            d2 -= prd32[2] * rintf(d2 * iprd32[2]);
            const float cut32 = ((float)ri + q.w + (float)skin) * 1.0001f + 1e-3f;
            if (d0 * d0 + d1 * d1 + d2 * d2 >= cut32 * cut32) continue;
            double d[3] = {xi[0] - x[j], xi[1] - x[n + j], xi[2] - x[2 * n + j]}, nimg[3];
            min_image(prd, iprd, d, nimg);
            const double rsq = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
            const double cut = (ri + rad[j]) + skin;
            if (rsq < cut * cut) {
                if (pj) {
                    pi[out] = i;
                    pj[out] = j;
                    ++out;
                }
                ++cnt;
            }
        }
    }
    if (act && !pj) count[i] = cnt;
}

// The same list by cells: atoms binned (positions wrapped) into a grid whose
// cells are at least the longest cut wide, at least three per axis, each atom
// tested against the 27 cells around it instead of every atom above it (31,250
// spheres: 2 x 3.1 ms for all pairs).  The order in which the atomics fill a
// cell does not show: a row's partners are sorted as they are written.
__device__ __forceinline__ int cell_axis(double x, double lo, double iprd, int g) {
    const double l = (x - lo) * iprd, f = l - floor(l);
    const int c = (int)(f * (double)g);
    return c < 0 ? 0 : (c < g ? c : g - 1);
}

struct Cells {
    int32_t *count, *start, *fill, *cell, *order;  // [m], [m + 1], [m] (the scan's tile totals first), [n], [n]
    float4* pos;                                   // [n] by cell: FP32 position and radius
};
Cells carve_cells(void* work, int n, int m) {
    char* p = static_cast<char*>(work);
    Cells c;
    c.count = reinterpret_cast<int32_t*>(p); p += align256((size_t)m * 4);
    c.start = reinterpret_cast<int32_t*>(p); p += align256(((size_t)m + 1) * 4);
    c.fill = reinterpret_cast<int32_t*>(p); p += align256((size_t)m * 4);
    c.cell = reinterpret_cast<int32_t*>(p); p += align256((size_t)n * 4);
    c.order = reinterpret_cast<int32_t*>(p); p += align256((size_t)n * 4);
    c.pos = reinterpret_cast<float4*>(p);
    return c;
}

__global__ void __launch_bounds__(128) k_cells_bin(int n, const double* __restrict__ x, const tmps_adj_rec* __restrict__ box,
                                                   int gx, int gy, int gz, Cells C) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int g[3] = {gx, gy, gz};
    int lin = 0;
#pragma unroll
    for (int c = 2; c >= 0; --c)
        lin = lin * g[c] + cell_axis(x[(size_t)c * n + i], box->lo[c], rcp64(box->prd[c]), g[c]);
    C.cell[i] = lin;
    atomicAdd(&C.count[lin], 1);
}

__global__ void __launch_bounds__(128) k_cells_fill(int n, const double* __restrict__ x, const double* __restrict__ rad,
                                                    Cells C) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int c = C.cell[i];
    const int p = C.start[c] + atomicAdd(&C.fill[c], 1);
    C.order[p] = i;
    C.pos[p] = make_float4((float)x[i], (float)x[n + i], (float)x[2 * n + i], (float)rad[i]);
}

__global__ void __launch_bounds__(64) k_pairs_cells(int n, const double* __restrict__ x, const double* __restrict__ rad,
                                                    const tmps_adj_rec* __restrict__ box, double skin, int gx, int gy,
                                                    int gz, Cells C, int32_t* __restrict__ count,
                                                    const int32_t* __restrict__ ibeg, int32_t* __restrict__ pi,
                                                    int32_t* __restrict__ pj) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    double prd[3], iprd[3];
    float prd32[3], iprd32[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        prd[c] = box->prd[c];
        iprd[c] = rcp64(prd[c]);
        prd32[c] = (float)prd[c];
        iprd32[c] = (float)iprd[c];
    }
    const int i = C.order[p];
    const float4 a = C.pos[p];
    const double xi[3] = {x[i], x[n + i], x[2 * n + i]}, ri = rad[i];
    const int lin = C.cell[i], cx = lin % gx, cy = (lin / gx) % gy, cz = lin / (gx * gy);
    const int beg = pj ? ibeg[i] : 0;
    int cnt = 0;
    for (int o = 0; o < 27; ++o) {
        int nx = cx + o % 3 - 1, ny = cy + (o / 3) % 3 - 1, nz = cz + o / 9 - 1;
        nx += nx < 0 ? gx : (nx >= gx ? -gx : 0);
        ny += ny < 0 ? gy : (ny >= gy ? -gy : 0);
        nz += nz < 0 ? gz : (nz >= gz ? -gz : 0);
        const int c = (nz * gy + ny) * gx + nx;
        for (int q = C.start[c]; q < C.start[c + 1]; ++q) {
            const int j = C.order[q];
            if (j <= i) continue;
            const float4 b = C.pos[q];
            float d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z;
            d0 -= prd32[0] * rintf(d0 * iprd32[0]);
            d1 -= prd32[1] * rintf(d1 * iprd32[1]);
            d2 -= prd32[2] * rintf(d2 * iprd32[2]);
            // an FP32 screen with a wide margin, then the exact FP64 test (neighbor.py:348-356)
            const float cut32 = (a.w + b.w + (float)skin) * 1.0001f + 1e-3f;
            if (d0 * d0 + d1 * d1 + d2 * d2 >= cut32 * cut32) continue;
            double d[3] = {xi[0] - x[j], xi[1] - x[n + j], xi[2] - x[2 * n + j]}, nimg[3];
            min_image(prd, iprd, d, nimg);
            const double rsq = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
            const double cut = (ri + rad[j]) + skin;
            if (!(rsq < cut * cut)) continue;
            if (pj) {
                int k = beg + cnt;
                for (; k > beg && pj[k - 1] > j; --k) pj[k] = pj[k - 1];
                pj[k] = j;
                pi[beg + cnt] = i;
            }
            ++cnt;
        }
    }
    if (!pj) count[i] = cnt;
}

__global__ void k_pair_map(int nold, const int32_t* __restrict__ opi, const int32_t* __restrict__ opj,
                           const int32_t* __restrict__ nibeg, const int32_t* __restrict__ npj, int32_t* __restrict__ map) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nold) return;
    const int i = opi[p], j = opj[p];
    int lo = nibeg[i], hi = nibeg[i + 1] - 1, r = -1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const int v = npj[mid];
        if (v == j) {
            r = mid;
            break;
        }
        if (v < j) lo = mid + 1;
        else hi = mid - 1;
    }
    map[p] = r;
}

__global__ void k_carry(int nold, int nnew, const int32_t* __restrict__ map, double* __restrict__ old_,
                        double* __restrict__ new_, int reverse) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nold) return;
    const int q = map[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (reverse) old_[(size_t)c * nold + p] = q >= 0 ? new_[(size_t)c * nnew + q] : 0.0;
        else if (q >= 0) new_[(size_t)c * nnew + q] = old_[(size_t)c * nold + p];
    }
}

// ---------------------------------------------------------------- forward

// First half of a step from S (remap == 0) or, inside a queued run, from the
// tape of the step before: its xh remapped from box `before` to `prev`.  The
// displacement check stamps q->hit (queued runs) or keeps the largest squared
// displacement (disp).
__global__ void __launch_bounds__(kBlk) k_initial(tmps_adj_sys S, double dt, tmps_adj_tape T, const double* xlast,
                                                  const tmps_adj_rec* before, const tmps_adj_rec* prev,
                                                  const double* __restrict__ xbuild, unsigned long long* disp, Queue* q,
                                                  int64_t step, double trig) {
    const int n = S.n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = i < n;
    // all but the new box is from kernels before the last: the half-kick, and the offset in the old box
    double v[3] = {0, 0, 0}, w[3] = {0, 0, 0}, x0[3] = {0, 0, 0}, xb[3] = {0, 0, 0};
    if (mine) {
        const double dtf = 0.5 * dt;
        const double m = S.mass[i], r = S.radius[i], I = inertia(m, r);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t k = (size_t)c * n + i;
            v[c] = S.v[k] + dtf * quot64(S.f[k], m);
            w[c] = S.w[k] + dtf * quot64(S.t[k], I);
            if (before) x0[c] = quot64(xlast[k] - before->lo[c], before->prd[c]);
            xb[c] = xbuild[k];
        }
    }
    enter();
    if (q) {
        const int64_t h = *(volatile const int64_t*)&q->hit;
        if (h != 0 && h != step) return;  // (another block of this step may have stamped it)
    }
    double dd = 0.0;
    if (mine) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t k = (size_t)c * n + i;
            // (S.x may be the last kernel's, the remap that ends a queued run)
            x0[c] = before ? prev->prd[c] * x0[c] + prev->lo[c] : S.x[k];
            const double x = x0[c] + dt * v[c];
            T.vh[k] = v[c];
            T.xh[k] = x;
            T.wh[k] = w[c];
            const double e = x - xb[c];
            dd += e * e;
        }
    }
    if (q) {
        if (__any_sync(0xffffffffu, dd > trig) && (threadIdx.x & 31) == 0) *(volatile int64_t*)&q->hit = step;
        return;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dd = fmax(dd, __shfl_down_sync(0xffffffffu, dd, o));
    // non-negative doubles order as their bit patterns
    if ((threadIdx.x & 31) == 0 && dd > 0.0) atomicMax(disp, (unsigned long long)__double_as_longlong(dd));
}

__device__ __forceinline__ void load_pair(const tmps_adj_sys& S, const double* xs, const double* vs, const double* ws,
                                          const double* prd, const double* iprd, int p, int i, int j, PairIn& in,
                                          double* nimg) {
    const int n = S.n;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        in.d[c] = xs[(size_t)c * n + i] - xs[(size_t)c * n + j];
        in.va[c] = vs[(size_t)c * n + i];
        in.vb[c] = vs[(size_t)c * n + j];
        in.wa[c] = ws[(size_t)c * n + i];
        in.wb[c] = ws[(size_t)c * n + j];
    }
    min_image(prd, iprd, in.d, nimg);
    in.ra = S.radius[i];
    in.rb = S.radius[j];
    in.ma = S.mass[i];
    in.mb = S.mass[j];
    (void)p;
}

// The pairs of a tile whose `in` holds, packed to the front of `list` in pair
// order (two warps, each two rounds of 32); returns their number.
__device__ __forceinline__ int pack_tile(const bool (&in)[kPairTile / kBlk], int* list /* [kPairTile] */,
                                         int* count /* [kPairTile / 32] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t b[kPairTile / kBlk];
#pragma unroll
    for (int u = 0; u < kPairTile / kBlk; ++u) {
        b[u] = __ballot_sync(0xffffffffu, in[u]);
        if (lane == 0) count[u * (kBlk / 32) + warp] = __popc(b[u]);
    }
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int w = 0; w < kPairTile / 32; ++w) {
#pragma unroll
        for (int u = 0; u < kPairTile / kBlk; ++u)
            if (w == u * (kBlk / 32) + warp && in[u]) list[total + __popc(b[u] & ((1u << lane) - 1u))] = u * kBlk + threadIdx.x;
        total += count[w];
    }
    __syncthreads();
    return total;
}

// Contacts of one pass: pair forces and torque terms into the workspace,
// history updated in place (the entering history recorded), virial partials.
// The tile's distances first; pairs out of contact are finished with zeros,
// the law runs over the rest with full warps.  The tile of block 2 g + h is
// warps h, h + 2, h + 4, h + 6 of group g (sum_groups): its threads' first
// round h and h + 4, their second h + 2 and h + 6.
__global__ void __launch_bounds__(kBlk) k_pairs(tmps_adj_sys S, Params P, int shearupdate, const double* xs,
                                                const double* vs, const double* ws, const tmps_adj_rec* __restrict__ box,
                                                double* __restrict__ sh_rec, uint8_t* __restrict__ mask_rec, Work W,
                                                const Queue* q) {
    __shared__ double svir[6][kPairTile], smem[6][kPairTile / 32];
    __shared__ int list[kPairTile], count[kPairTile / 32];
    const int n = S.n, np = S.npairs;
    double prd[3], iprd[3], nimg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        prd[c] = box->prd[c];
        iprd[c] = rcp64(prd[c]);
    }
    // the pair of the tile's entry e = 64 round + thread
    const int group = (int)(blockIdx.x >> 1) * kSum, h = blockIdx.x & 1;
    auto pair_at = [&](int e) { return group + 32 * (h + 2 * (e >> 6) + 4 * ((e >> 5) & 1)) + (e & 31); };
    int pi[kPairTile / kBlk], pj[kPairTile / kBlk];
    double radsum_[kPairTile / kBlk];
#pragma unroll
    for (int u = 0; u < kPairTile / kBlk; ++u) {
        const int p = pair_at(u * kBlk + threadIdx.x);
        pi[u] = p < np ? S.pi[p] : 0;
        pj[u] = p < np ? S.pj[p] : 0;
        radsum_[u] = S.radius[pi[u]] + S.radius[pj[u]];
    }
    enter();
    if (halted(q)) return;
    bool in_[kPairTile / kBlk];
#pragma unroll
    for (int u = 0; u < kPairTile / kBlk; ++u) {
        const int p = pair_at(u * kBlk + threadIdx.x);
        in_[u] = false;
#pragma unroll
        for (int c = 0; c < 6; ++c) svir[c][u * kBlk + threadIdx.x] = 0.0;
        if (p < np) {
            const int i = pi[u], j = pj[u];
            double d[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) d[c] = xs[(size_t)c * n + i] - xs[(size_t)c * n + j];
            min_image(prd, iprd, d, nimg);
            const double rsq = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2];
            const double radsum = radsum_[u];
            in_[u] = rsq < radsum * radsum && rsq > 1e-28;
            if (!in_[u]) {
                mask_rec[p] = 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    sh_rec[(size_t)c * np + p] = S.shear[(size_t)c * np + p];
                    S.shear[(size_t)c * np + p] = 0.0;
                }
            }
        }
    }
    const int total = pack_tile(in_, list, count);
    for (int k = threadIdx.x; k < total; k += kBlk) {
        const int p = pair_at(list[k]);
        PairIn in;
        load_pair(S, xs, vs, ws, prd, iprd, p, S.pi[p], S.pj[p], in, nimg);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            in.sh[c] = S.shear[(size_t)c * np + p];
            sh_rec[(size_t)c * np + p] = in.sh[c];
        }
        PairOut o;
        PairTape t;
        int mask;
        pair_forward(P, shearupdate, in, -1, o, t, &mask);
        mask_rec[p] = (uint8_t)mask;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            S.shear[(size_t)c * np + p] = o.sh[c];
            W.fp[(size_t)c * np + p] = o.F[c];
            W.tp[(size_t)c * np + p] = o.tor[c];
        }
        const int e = list[k];
        svir[0][e] = in.d[0] * o.F[0];
        svir[1][e] = in.d[1] * o.F[1];
        svir[2][e] = in.d[2] * o.F[2];
        svir[3][e] = in.d[0] * o.F[1];
        svir[4][e] = in.d[0] * o.F[2];
        svir[5][e] = in.d[1] * o.F[2];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPairTile / kBlk; ++u) {
        const int e = u * kBlk + threadIdx.x;
        const double v[6] = {svir[0][e], svir[1][e], svir[2][e], svir[3][e], svir[4][e], svir[5][e]};
        const double t = warp_sum6_halving(v);  // lane >> 2 is the component
        const int c = (threadIdx.x & 31) >> 2;
        if ((threadIdx.x & 3) == 0 && c < 6) smem[c][e >> 5] = t;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const double* w = smem[threadIdx.x];
        W.partw[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = (w[0] + w[1]) + (w[2] + w[3]);
    }
}

// Per-atom force and torque from the pairs in contact (as i: +F, then as j:
// -F; the torque term times -r either way), then the second half-kick (final =
// 1) and the kinetic partials m v v.  Blocks 4 g .. 4 g + 3 take warps 0 and 4,
// 2 and 6, 1 and 5, 3 and 7 of group g (sum_groups).
__global__ void __launch_bounds__(kBlk) k_gather(tmps_adj_sys S, double dt, int final_, const double* __restrict__ vh,
                                                 const double* __restrict__ wh, double* __restrict__ ft,
                                                 double* __restrict__ tt, const uint8_t* mask, Work W, const Queue* q) {
    __shared__ double smem[6][kBlk / 32];
    const int n = S.n, np = S.npairs;
    const int quarter = blockIdx.x & 3;
    const int a = (int)(blockIdx.x >> 2) * kSum +
                  32 * (((quarter & 1) << 1 | quarter >> 1) + 4 * (int)(threadIdx.x >> 5)) + (threadIdx.x & 31);
    double kin[6] = {0, 0, 0, 0, 0, 0};
    int i0 = 0, ni = 0, j0 = 0, nj = 0;
    double ra = 0.0, m = 1.0, I = 1.0, im = 1.0, iI = 1.0, vh0[3] = {0, 0, 0}, wh0[3] = {0, 0, 0};
    if (a < n) {
        i0 = S.ibeg[a];
        ni = S.ibeg[a + 1] - i0;
        j0 = S.jbeg[a];
        nj = S.jbeg[a + 1] - j0;
        ra = S.radius[a];
        m = S.mass[a];
        I = inertia(m, ra);
        im = near_rcp64(m);  // for div_by
        iI = near_rcp64(I);
        if (final_)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                vh0[c] = vh[(size_t)c * n + a];
                wh0[c] = wh[(size_t)c * n + a];
            }
    }
    // the pair of entry k: first the atom's pairs as i, then as j
    auto pair_of = [&](int k) { return k < ni ? i0 + k : S.jlist[j0 + k - ni]; };
    int p0[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) p0[u] = u < ni + nj ? pair_of(u) : 0;
    enter();
    if (halted(q)) return;
    if (a < n) {
        double F[3] = {0, 0, 0}, Tq[3] = {0, 0, 0};
        // four pairs' masks and terms in flight together (a term is used where the mask says contact)
        for (int k0 = 0; k0 < ni + nj; k0 += 4) {
            int p[4];
            uint8_t on[4];
            double f[4][6];
#pragma unroll
            for (int u = 0; u < 4; ++u) p[u] = k0 == 0 ? p0[u] : (k0 + u < ni + nj ? pair_of(k0 + u) : 0);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                on[u] = k0 + u < ni + nj ? mask[p[u]] : 0;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    f[u][c] = W.fp[(size_t)c * np + p[u]];
                    f[u][3 + c] = W.tp[(size_t)c * np + p[u]];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!on[u]) continue;
                const bool first = k0 + u < ni;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    F[c] += first ? f[u][c] : -f[u][c];
                    Tq[c] += -ra * f[u][3 + c];
                }
            }
        }
        const double dtf = 0.5 * dt;
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t k = (size_t)c * n + a;
            S.f[k] = F[c];
            S.t[k] = Tq[c];
            if (ft) {
                ft[k] = F[c];
                tt[k] = Tq[c];
            }
            if (final_) {
                v[c] = vh0[c] + dtf * div_by(F[c], m, im);
                S.v[k] = v[c];
                S.w[k] = wh0[c] + dtf * div_by(Tq[c], I, iI);
            }
        }
        if (final_) {
            kin[0] = (m * v[0]) * v[0];
            kin[1] = (m * v[1]) * v[1];
            kin[2] = (m * v[2]) * v[2];
            kin[3] = (m * v[0]) * v[1];
            kin[4] = (m * v[0]) * v[2];
            kin[5] = (m * v[1]) * v[2];
        }
    }
    if (!final_) return;
    const double t = warp_sum6_halving(kin);  // lane >> 2 is the component
    const int c = (threadIdx.x & 31) >> 2;
    if ((threadIdx.x & 3) == 0 && c < 6) smem[c][threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x < 6)
        W.partk[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = smem[threadIdx.x][0] + smem[threadIdx.x][1];
}

// The servo rate of a pressure axis: gain, normalize/pressure, max/rate
// (_limit_rate_device, deform_pressure.py:583-596).  Sets *clamped when
// max/rate (or a zero target under normalize) fixed the value.
__device__ double servo_rate(const tmps_adj_servo& sv, int d, double pd, bool* clamped) {
    double out = sv.pgain[d] * (pd - sv.ptarget[d]);
    *clamped = false;
    if (sv.normalize == 1) {
        if (sv.ptarget[d] == 0.0) {
            if (out != 0.0) {
                out = sv.max_rate * (out > 0.0 ? 1.0 : -1.0);
                *clamped = true;
            }
        } else {
            out = out / fabs(sv.ptarget[d]);
        }
    }
    if (sv.max_rate != 0.0 && fabs(out) > sv.max_rate) {
        out = sv.max_rate * (out > 0.0 ? 1.0 : -1.0);
        *clamped = true;
    }
    return out;
}

__device__ void coupled(int couple, const double* P, double* p) {
    p[0] = P[0];
    p[1] = P[1];
    p[2] = P[2];
    if (couple == 1) {
        const double s = (P[0] + P[1] + P[2]) / 3.0;
        p[0] = p[1] = p[2] = s;
    } else if (couple == 2) {
        const double m = 0.5 * (P[0] + P[1]);
        p[0] = p[1] = m;
    } else if (couple == 3) {
        const double m = 0.5 * (P[1] + P[2]);
        p[1] = p[2] = m;
    } else if (couple == 4) {
        const double m = 0.5 * (P[0] + P[2]);
        p[0] = p[2] = m;
    }
}

// Virial total, pressure tensor, deviatoric stress, the servo's new box.
__global__ void __launch_bounds__(kOne) k_servo(tmps_adj_servo sv, double dt, int64_t step, const tmps_adj_rec* prev,
                                                tmps_adj_rec* next, int ngP, int ngA, Work W, Queue* q) {
    __shared__ double sw[6], sk[6];
    sum_groups<2>(W.partw, ngP, sw, 0);
    tmps_adj_rec r;
    double vol = 1.0, ivol = 1.0;
    if (threadIdx.x == 0) {
        r = *prev;
        vol = (r.prd[0] * r.prd[1]) * r.prd[2];
        ivol = near_rcp64(vol);  // for div_by
    }
    enter();
    if (halted(q)) return;
    sum_groups<4>(W.partk, ngA, sk, 6);
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (q) q->done = step;
    double Pt[6];
    for (int c = 0; c < 6; ++c) {
        r.w[c] = sw[c] + sk[c];
        Pt[c] = div_by(r.w[c], vol, ivol);
    }
    r.q = Pt[2] - 0.5 * (Pt[0] + Pt[1]);
    r.elapsed = (double)step * dt;
    double p[3];
    coupled(sv.couple, Pt, p);
    r.clamp = 0;
    for (int d = 0; d < 3; ++d) {
        const double lo_s = sv.lo_start[d], hi_s = sv.hi_start[d];
        double lo, hi;
        if (sv.style[d] == 1) {
            const double shift = ((0.5 * r.elapsed) * sv.rate[d]) * (hi_s - lo_s);
            lo = lo_s - shift;
            hi = hi_s + shift;
        } else if (sv.style[d] == 8) {
            bool cl;
            const double rate = servo_rate(sv, d, p[d], &cl);
            if (cl) r.clamp |= 1 << d;
            r.cum[d] += (dt * rate) * r.prd[d];
            lo = lo_s - 0.5 * r.cum[d];
            hi = hi_s + 0.5 * r.cum[d];
        } else {
            continue;  // style none: the box stays as it is
        }
        r.lo[d] = lo;
        r.prd[d] = hi - lo;
    }
    *next = r;
}

__global__ void __launch_bounds__(kBlk) k_remap(int n, const double* __restrict__ xh, const tmps_adj_rec* prev,
                                                const tmps_adj_rec* next, double* __restrict__ x, const Queue* q) {
    enter();
    if (halted(q)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const size_t k = (size_t)c * n + i;
        const double lam = quot64(xh[k] - prev->lo[c], prev->prd[c]);
        x[k] = next->prd[c] * lam + next->lo[c];
    }
}

// ---------------------------------------------------------------- reverse

// The parameter and image partials of step `step` + 1's contact pass (reduce =
// 1), then the reverse of step `step`'s servo and pressure (servo = 1): box adjoints (slot of record n =
// step - 1 and of record n + 1 by parity), dL/d(virial total) into W.wbar.
__global__ void __launch_bounds__(kOne) k_b_servo(tmps_adj_servo sv, double dt, int64_t step, const tmps_adj_rec* prev,
                                                  const tmps_adj_rec* next, double qbar, int nbA, int nbP, int reduce,
                                                  int servo, int slot, tmps_adj_bar B, Work W) {
    __shared__ double s[6], g[8], box[18], par[5], wbar[6];
    __shared__ double sPt[6], sratio[3], srate[3];
    const int tid = threadIdx.x;
    // what the records alone give, and the accumulated adjoints, before the wait
    if (tid < 18) box[tid] = B.box[tid];
    if (tid >= 32 && tid < 37) par[tid - 32] = B.params[tid - 32];
    if (tid == kOne - 32 && servo) {
        const double vol = (prev->prd[0] * prev->prd[1]) * prev->prd[2];
        double Pt[6], p[3];
        for (int c = 0; c < 6; ++c) sPt[c] = Pt[c] = quot64(next->w[c], vol);
        coupled(sv.couple, Pt, p);
        for (int d = 0; d < 3; ++d) {
            bool cl;
            sratio[d] = quot64(next->prd[d], prev->prd[d]);
            srate[d] = sv.style[d] == 8 ? servo_rate(sv, d, p[d], &cl) : 0.0;
        }
    }
    double prd[3] = {1, 1, 1}, vol = 1.0, ivol = 1.0;
    int clamp = 0;
    if (tid == 0 && servo) {
        for (int d = 0; d < 3; ++d) prd[d] = prev->prd[d];
        vol = (prd[0] * prd[1]) * prd[2];
        ivol = near_rcp64(vol);  // for div_by
        clamp = next->clamp;
    }
    enter();
    if (servo) sum_partials<6>(W.partk, nbA, s, 0);
    if (reduce) sum_partials<8>(W.partg, nbP, g, 6);
    __syncthreads();
    if (tid == 0) {
        if (reduce) {
            for (int c = 0; c < 5; ++c) par[c] += g[c];
            for (int c = 0; c < 3; ++c) box[9 * slot + 3 + c] += g[5 + c];
        }
        if (servo) {
            const int n = (int)((step - 1) & 1);
            double* const bn = box + 9 * n;          // record step - 1: lo 0..2, prd 3..5, cum 6..8
            double* const bn1 = box + 9 * (1 - n);   // record step
            double pb[3] = {0, 0, 0}, Pb[6] = {0, 0, 0, 0, 0, 0};
            for (int d = 0; d < 3; ++d) {
                const double ratio = sratio[d];
                // remap
                bn1[d] += s[d];
                bn1[3 + d] += s[3 + d];
                bn[d] -= s[d] * ratio;
                bn[3 + d] -= s[3 + d] * ratio;
                if (sv.style[d] != 8) continue;
                // record step's box from its cumulative shift: lo = lo_s - cum / 2, prd = L + cum
                const double cumb = bn1[6 + d] + bn1[3 + d] - 0.5 * bn1[d];
                // cum' = cum + (dt rate) prd
                bn[6 + d] += cumb;
                bn[3 + d] += cumb * dt * srate[d];
                if (!((clamp >> d) & 1)) {
                    double rb = cumb * dt * prd[d] * sv.pgain[d];
                    if (sv.normalize == 1) rb = rb / fabs(sv.ptarget[d]);
                    pb[d] += rb;
                }
            }
            for (int c = 0; c < 9; ++c) bn1[c] = 0.0;
            // couple
            if (sv.couple == 1) {
                const double m = (pb[0] + pb[1] + pb[2]) / 3.0;
                Pb[0] = Pb[1] = Pb[2] = m;
            } else if (sv.couple == 2) {
                Pb[0] = Pb[1] = 0.5 * (pb[0] + pb[1]);
                Pb[2] = pb[2];
            } else if (sv.couple == 3) {
                Pb[1] = Pb[2] = 0.5 * (pb[1] + pb[2]);
                Pb[0] = pb[0];
            } else if (sv.couple == 4) {
                Pb[0] = Pb[2] = 0.5 * (pb[0] + pb[2]);
                Pb[1] = pb[1];
            } else {
                Pb[0] = pb[0];
                Pb[1] = pb[1];
                Pb[2] = pb[2];
            }
            // deviatoric stress q = Pzz - (Pxx + Pyy) / 2
            Pb[2] += qbar;
            Pb[0] -= 0.5 * qbar;
            Pb[1] -= 0.5 * qbar;
            // P = W / vol
            double volb = 0.0;
            for (int c = 0; c < 6; ++c) {
                wbar[c] = div_by(Pb[c], vol, ivol);
                volb -= div_by(Pb[c] * sPt[c], vol, ivol);
            }
            bn[3] += volb * prd[1] * prd[2];
            bn[4] += volb * prd[0] * prd[2];
            bn[5] += volb * prd[0] * prd[1];
        }
    }
    __syncthreads();
    if (tid < 18) B.box[tid] = box[tid];
    if (tid >= 32 && tid < 37) B.params[tid - 32] = par[tid - 32];
    if (servo && tid >= 64 && tid < 70) W.wbar[tid - 64] = wbar[tid - 64];
}

// Reverse of the second half-kick and of the kinetic virial term.
__global__ void __launch_bounds__(kBlk) k_b_final(tmps_adj_sys S, double dt, tmps_adj_tape T, tmps_adj_bar B, Work W) {
    const int n = S.n;
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = a < n;
    double m = 1.0, r = 1.0, I = 1.0, im = 1.0, iI = 1.0, v[3] = {0, 0, 0}, vb[3] = {0, 0, 0}, f[3] = {0, 0, 0}, fb[3] = {0, 0, 0};
    double mb = 0.0, Ib = 0.0, mass0 = 0.0, rad0 = 0.0;
    const double dtf = 0.5 * dt;
    if (mine) {
        m = S.mass[a];
        r = S.radius[a];
        I = inertia(m, r);
        im = near_rcp64(m);  // for div_by
        iI = near_rcp64(I);
        mass0 = B.mass[a];
        rad0 = B.radius[a];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t k = (size_t)c * n + a;
            f[c] = T.f[k];
            v[c] = T.vh[k] + dtf * div_by(f[c], m, im);
            vb[c] = B.v[k];
            fb[c] = B.f[k];
            // w = wh + dtf t / I
            const double wb = dtf * B.w[k];
            B.t[k] += div_by(wb, I, iI);
            Ib -= div_by(wb * T.t[k], I * I, iI * iI);
        }
    }
    enter();
    if (!mine) return;
    double wb[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) wb[c] = W.wbar[c];
    // kinetic m v_a v_b
    vb[0] += m * (2.0 * wb[0] * v[0] + wb[3] * v[1] + wb[4] * v[2]);
    vb[1] += m * (2.0 * wb[1] * v[1] + wb[3] * v[0] + wb[5] * v[2]);
    vb[2] += m * (2.0 * wb[2] * v[2] + wb[4] * v[0] + wb[5] * v[1]);
    mb = wb[0] * v[0] * v[0] + wb[1] * v[1] * v[1] + wb[2] * v[2] * v[2] + wb[3] * v[0] * v[1] +
         wb[4] * v[0] * v[2] + wb[5] * v[1] * v[2];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const size_t k = (size_t)c * n + a;
        // v = vh + dtf f / m
        const double kb = dtf * vb[c];
        B.v[k] = vb[c];
        B.f[k] = fb[c] + div_by(kb, m, im);
        mb -= div_by(kb * f[c], m * m, im * im);
    }
    B.mass[a] = mass0 + (mb + Ib * 0.4 * r * r);
    B.radius[a] = rad0 + Ib * 0.8 * m * r;
}

// Reverse of the contact pass: per pair in contact, recompute under the
// recorded mask, then the reverse; per-pair adjoints for the gather, the
// entering history's adjoint in place, parameter and image partials.
//
// kPerSM: resident blocks asked of the compiler.  Four leave it all 255
// registers; five have 168 and spill.  Five pay where they take up most of a
// second wave of four and no more (run_b_pairs).  Gradient of 60 steps, four
// against five, by the tiles (608 and 760 a wave): 46 6.26 and 6.56 ms, 180
// 7.56 and 7.87, 401 10.46 and 10.20, 602 11.08 and 12.16, 803 14.10 and 13.24,
// 1,201 15.18 and 17.30, 1,606 21.28 and 21.62, 3,212 38.5 and 39.4.
template <int kPerSM>
__global__ void __launch_bounds__(kBlk, kPerSM) k_b_pairs(tmps_adj_sys S, Params P, int shearupdate, const double* xs,
                                                  const double* vs, const double* ws, const double* __restrict__ sh_rec,
                                                  const uint8_t* __restrict__ mask_rec,
                                                  const tmps_adj_rec* __restrict__ box, const double* __restrict__ wbar,
                                                  tmps_adj_bar B, Work W) {
    __shared__ double smem[8 * (kBlk / 32)];
    __shared__ int list[kPairTile], count[kPairTile / 32];
    // (only the adjoints of the forces are the last kernel's: the contacts are recomputed before the wait)
    const int n = S.n, np = S.npairs;
    double prd[3], iprd[3], nimg[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        prd[c] = box->prd[c];
        iprd[c] = rcp64(prd[c]);
    }
    bool waited = false;
    bool in_[kPairTile / kBlk];
#pragma unroll
    for (int u = 0; u < kPairTile / kBlk; ++u) {
        const int p = blockIdx.x * kPairTile + u * kBlk + threadIdx.x;
        in_[u] = p < np && mask_rec[p] != 0;
        // out of contact: no force, and the history that leaves is zero whatever entered
        if (p < np && !in_[u]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) B.shear[(size_t)c * np + p] = 0.0;
        }
    }
    const int total = pack_tile(in_, list, count);
    double part[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int k = threadIdx.x; k < total; k += kBlk) {
        const int p = blockIdx.x * kPairTile + list[k];
        const int i = S.pi[p], j = S.pj[p];
        PairIn in;
        load_pair(S, xs, vs, ws, prd, iprd, p, i, j, in, nimg);
#pragma unroll
        for (int c = 0; c < 3; ++c) in.sh[c] = sh_rec[(size_t)c * np + p];
        PairOut o;
        PairTape t;
        int mask;
        const int rec = mask_rec[p];
        pair_forward(P, shearupdate, in, rec, o, t, &mask);
        if (!waited) enter();
        waited = true;
        PairBar b;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            b.fa[c] = B.f[(size_t)c * n + i];
            b.fb[c] = B.f[(size_t)c * n + j];
            b.ta[c] = B.t[(size_t)c * n + i];
            b.tb[c] = B.t[(size_t)c * n + j];
            b.sh[c] = B.shear[(size_t)c * np + p];
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) b.w[c] = wbar ? wbar[c] : 0.0;
        PairGrad g;
        pair_reverse(P, shearupdate, rec, in, o, t, b, g);
        double* G = W.gp;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            B.shear[(size_t)c * np + p] = g.sh[c];
            G[(size_t)c * np + p] = g.d[c];
            G[(size_t)(3 + c) * np + p] = g.vrel[c];
            G[(size_t)(6 + c) * np + p] = g.wa[c];
            G[(size_t)(9 + c) * np + p] = g.wb[c];
        }
        G[(size_t)12 * np + p] = g.ra;
        G[(size_t)13 * np + p] = g.rb;
        G[(size_t)14 * np + p] = g.ma;
        G[(size_t)15 * np + p] = g.mb;
        part[0] += g.kn;
        part[1] += g.kt;
        part[2] += g.gamman;
        part[3] += g.gammat;
        part[4] += g.xmu;
        // d = xa - xb - nimg prd
#pragma unroll
        for (int c = 0; c < 3; ++c) part[5 + c] -= nimg[c] * g.d[c];
    }
    if (!waited) enter();
    block_sum<8, kBlk>(part, smem);
    if (threadIdx.x == 0) {
        const int nb = gridDim.x;
#pragma unroll
        for (int c = 0; c < 8; ++c) W.partg[(size_t)c * nb + blockIdx.x] = part[c];
    }
}

// Per atom: the sums of the pairs' adjoints (as i, then as j) and the reverse
// of the first half-kick and the drift of a step (gather = 1: leaves the
// adjoint of the state before it, and of the forces it started from; kick = 0:
// the sums alone), then the reverse of the remap that ended the step before
// (xh != NULL): x' = prd' (xh - lo) / prd + lo', the adjoint of xh in place and
// the partial sums of x'bar and x'bar lam per dimension for the box adjoints.
__global__ void __launch_bounds__(kBlk) k_b_atoms(tmps_adj_sys S, double dt, int gather, int kick,
                                                  const uint8_t* mask, const double* __restrict__ fprev,
                                                  const double* __restrict__ tprev, const double* __restrict__ xh,
                                                  const tmps_adj_rec* prev, const tmps_adj_rec* next, tmps_adj_bar B,
                                                  Work W) {
    __shared__ double smem[6 * (kBlk / 32)];
    const int n = S.n, np = S.npairs;
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = a < n;
    double s[6] = {0, 0, 0, 0, 0, 0};
    // everything but the pairs' adjoints before the wait
    int i0 = 0, ni = 0, j0 = 0, nj = 0;
    double m = 1.0, r = 1.0, I = 1.0, im = 1.0, iI = 1.0, mass0 = 0.0, rad0 = 0.0;
    double x0[3] = {0, 0, 0}, v0[3] = {0, 0, 0}, w0[3] = {0, 0, 0}, fp[3] = {0, 0, 0}, tp[3] = {0, 0, 0}, lam[3] = {0, 0, 0},
           scale[3] = {1, 1, 1};
    if (mine) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const size_t k = (size_t)c * n + a;
            x0[c] = B.x[k];
            if (xh) {
                lam[c] = quot64(xh[k] - prev->lo[c], prev->prd[c]);
                scale[c] = quot64(next->prd[c], prev->prd[c]);
            }
            if (gather) {
                v0[c] = B.v[k];
                w0[c] = B.w[k];
                if (kick) {
                    fp[c] = fprev[k];
                    tp[c] = tprev[k];
                }
            }
        }
        if (gather) {
            i0 = S.ibeg[a];
            ni = S.ibeg[a + 1] - i0;
            j0 = S.jbeg[a];
            nj = S.jbeg[a + 1] - j0;
            m = S.mass[a];
            r = S.radius[a];
            I = inertia(m, r);
            im = near_rcp64(m);  // for div_by
            iI = near_rcp64(I);
            mass0 = B.mass[a];
            rad0 = B.radius[a];
        }
    }
    auto pair_of = [&](int k) { return k < ni ? i0 + k : S.jlist[j0 + k - ni]; };
    constexpr int kPer = 3;
    int p0[kPer];
    uint8_t on0[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        p0[u] = u < ni + nj ? pair_of(u) : 0;
        on0[u] = u < ni + nj ? mask[p0[u]] : 0;
    }
    enter();
    if (mine) {
        if (gather) {
            const double* G = W.gp;
            double xb[3] = {0, 0, 0}, vb[3] = {0, 0, 0}, wb[3] = {0, 0, 0}, rb = 0.0, mb = 0.0;
            // a few pairs' adjoints in flight together
            for (int k0 = 0; k0 < ni + nj; k0 += kPer) {
                int p[kPer];
                uint8_t on[kPer];
                double g[kPer][11];
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    p[u] = k0 == 0 ? p0[u] : (k0 + u < ni + nj ? pair_of(k0 + u) : 0);
                    on[u] = k0 == 0 ? on0[u] : (k0 + u < ni + nj ? mask[p[u]] : 0);
                }
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const bool first = k0 + u < ni;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        g[u][c] = G[(size_t)c * np + p[u]];
                        g[u][3 + c] = G[(size_t)(3 + c) * np + p[u]];
                        g[u][6 + c] = G[(size_t)((first ? 6 : 9) + c) * np + p[u]];
                    }
                    g[u][9] = G[(size_t)(first ? 12 : 13) * np + p[u]];
                    g[u][10] = G[(size_t)(first ? 14 : 15) * np + p[u]];
                }
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    if (!on[u]) continue;
                    const bool first = k0 + u < ni;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        xb[c] += first ? g[u][c] : -g[u][c];
                        vb[c] += first ? g[u][3 + c] : -g[u][3 + c];
                        wb[c] += g[u][6 + c];
                    }
                    rb += g[u][9];
                    mb += g[u][10];
                }
            }
            const double dtf = 0.5 * dt;
            double Ib = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const size_t k = (size_t)c * n + a;
                x0[c] += xb[c];
                const double v1 = v0[c] + vb[c], w1 = w0[c] + wb[c];
                B.w[k] = w1;
                if (kick) {
                    // x = x0 + dt vh; vh = v0 + dtf f / m; wh = w0 + dtf t / I
                    const double vhb = v1 + dt * x0[c];
                    const double fb = dtf * vhb, tb = dtf * w1;
                    B.v[k] = vhb;
                    B.f[k] = div_by(fb, m, im);
                    mb -= div_by(fb * fp[c], m * m, im * im);
                    B.t[k] = div_by(tb, I, iI);
                    Ib -= div_by(tb * tp[c], I * I, iI * iI);
                } else {
                    B.v[k] = v1;
                }
                if (!xh) B.x[k] = x0[c];
            }
            B.mass[a] = mass0 + (mb + Ib * 0.4 * r * r);
            B.radius[a] = rad0 + (rb + Ib * 0.8 * m * r);
        }
        if (xh) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s[c] = x0[c];
                s[3 + c] = x0[c] * lam[c];
                B.x[(size_t)c * n + a] = x0[c] * scale[c];
            }
        }
    }
    if (!xh) return;
    const double tot = block_sum6_halving<kBlk>(s, 0.0, true, smem);
    if (threadIdx.x < 6) W.partk[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = tot;
}

bool ok() { return cudaPeekAtLastError() == cudaSuccess; }

bool sys_ok(const tmps_adj_sys* s) {
    return s && s->n >= 0 && s->npairs >= 0 && s->x && s->v && s->w && s->f && s->t && s->radius && s->mass &&
           (s->npairs == 0 || (s->shear && s->pi && s->pj)) && s->ibeg && s->jbeg && (s->npairs == 0 || s->jlist);
}

// The launches of one call: with programmatic stream serialization (see enter),
// but for the first, which starts once all that was queued before the call has
// completed; counted.
struct Chain {
    cudaStream_t stream;
    bool first = true;

    template <typename... P, typename... A>
    void run(void (*kernel)(P...), int grid, int block, A&&... args) {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = first ? 0 : 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3((unsigned)block);
        cfg.stream = stream;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
        first = false;
        note_launches(1);
    }
    // the next launch reads before its wait what the one before it writes
    void join() { first = true; }
    // The contact pass's reverse at the residency its number of tiles wants: with five blocks an SM
    // between one wave of four and one and a half.
    template <typename... A>
    void run_b_pairs(int tiles, A&&... args) {
        static const int wave = wave_blocks(k_b_pairs<4>, kBlk);
        if (tiles <= wave || tiles > wave + wave / 2) run(k_b_pairs<4>, tiles, kBlk, std::forward<A>(args)...);
        else run(k_b_pairs<5>, tiles, kBlk, std::forward<A>(args)...);
    }
};

// The tape of the k-th step of a run whose tapes lie atom_stride doubles (atom
// arrays) and pair_stride pairs apart (0: one tape, overwritten).
tmps_adj_tape tape_at(const tmps_adj_tape& t, int64_t atom_stride, int64_t pair_stride, int64_t k) {
    tmps_adj_tape o = t;
    o.xh += k * atom_stride;
    o.vh += k * atom_stride;
    o.wh += k * atom_stride;
    o.f += k * atom_stride;
    o.t += k * atom_stride;
    o.shear += 3 * k * pair_stride;
    o.mask += k * pair_stride;
    return o;
}

// Contacts, second half-kick, pressure and servo of a step.
int rest_of_step(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_servo* sv, const tmps_adj_tape& t,
                 tmps_adj_rec* d_rec, int64_t step, const Work& W, Queue* q, Chain& ch) {
    const int nbA = blocks_a(s->n), nbP = blocks_p(s->npairs);
    const tmps_adj_rec* prev = d_rec + (step - 1);
    if (s->npairs > 0) {
        ch.run(k_pairs, nbP, kBlk, *s, to_params(*p), 1, (const double*)t.xh, (const double*)t.vh, (const double*)t.wh,
            prev, t.shear, t.mask, W, (const Queue*)q);
    } else if (cudaMemsetAsync(W.partw, 0, sizeof(double) * 6 * nbP, ch.stream) != cudaSuccess) {
        return TMPS_ERR_CUDA;
    }
    if (s->n > 0) {
        ch.run(k_gather, nbA, kBlk, *s, p->dt, 1, (const double*)t.vh, (const double*)t.wh, t.f, t.t,
            (const uint8_t*)t.mask, W, (const Queue*)q);
    } else if (cudaMemsetAsync(W.partk, 0, sizeof(double) * 6 * nbA, ch.stream) != cudaSuccess) {
        return TMPS_ERR_CUDA;
    }
    ch.run(k_servo, 1, kOne, *sv, p->dt, step, prev, d_rec + step, grid_for(s->npairs, kSum), grid_for(s->n, kSum), W, q);
    return TMPS_OK;
}

}  // namespace

extern "C" {

int64_t tmps_adj_workspace_bytes(int32_t n, int32_t npairs) {
    if (n < 0 || npairs < 0) return -1;
    return (int64_t)work_bytes(n, npairs);
}

int tmps_adj_pairs(int32_t n, const double* d_x, const double* d_radius, const tmps_adj_rec* d_box, double skin,
                   int32_t* d_count, const int32_t* d_ibeg, int32_t* d_pi, int32_t* d_pj, void* stream) {
    if (n < 0 || !d_x || !d_radius || !d_box || !(skin >= 0.0)) return TMPS_ERR_BAD_ARG;
    if (!d_pj && !d_count) return TMPS_ERR_BAD_ARG;
    if (d_pj && (!d_ibeg || !d_pi)) return TMPS_ERR_BAD_ARG;
    if (n == 0) return TMPS_OK;
    k_pairs_build<<<grid_for(n, 128), 128, 0, (cudaStream_t)stream>>>(n, d_x, d_radius, d_box, skin, d_count, d_ibeg,
                                                                      d_pi, d_pj);
    note_launches(1);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int64_t tmps_adj_cells_bytes(int32_t n, int32_t ncell) {
    if (n < 0 || ncell < 0) return -1;
    return (int64_t)(3 * align256(((size_t)ncell + 1) * 4) + 2 * align256((size_t)n * 4) + align256((size_t)n * 16));
}

int tmps_adj_pairs_cells(int32_t n, const double* d_x, const double* d_radius, const tmps_adj_rec* d_box, double skin,
                         int32_t gx, int32_t gy, int32_t gz, void* work, int32_t* d_count, const int32_t* d_ibeg,
                         int32_t* d_pi, int32_t* d_pj, void* stream) {
    if (n < 0 || !d_x || !d_radius || !d_box || !(skin >= 0.0) || !work) return TMPS_ERR_BAD_ARG;
    if (gx < 3 || gy < 3 || gz < 3 || (int64_t)gx * gy * gz > (1 << 28)) return TMPS_ERR_BAD_ARG;
    if (!d_pj && !d_count) return TMPS_ERR_BAD_ARG;
    if (d_pj && (!d_ibeg || !d_pi)) return TMPS_ERR_BAD_ARG;
    if (n == 0) return TMPS_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const int m = gx * gy * gz;
    const Cells C = carve_cells(work, n, m);
    if (!d_pj) {
        // bins for both calls
        if (cudaMemsetAsync(C.count, 0, (size_t)m * 4, s) != cudaSuccess) return TMPS_ERR_CUDA;
        k_cells_bin<<<grid_for(n, 128), 128, 0, s>>>(n, d_x, d_box, gx, gy, gz, C);
        exclusive_scan(C.count, C.start, C.fill, m, s);
        if (cudaMemsetAsync(C.fill, 0, (size_t)m * 4, s) != cudaSuccess) return TMPS_ERR_CUDA;
        k_cells_fill<<<grid_for(n, 128), 128, 0, s>>>(n, d_x, d_radius, C);
        note_launches(4);
    }
    k_pairs_cells<<<grid_for(n, 64), 64, 0, s>>>(n, d_x, d_radius, d_box, skin, gx, gy, gz, C, d_count, d_ibeg, d_pi,
                                                 d_pj);
    note_launches(1);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_pair_map(int32_t nold, const int32_t* d_old_pi, const int32_t* d_old_pj, const int32_t* d_new_ibeg,
                      const int32_t* d_new_pj, int32_t* d_map, void* stream) {
    if (nold < 0 || (nold > 0 && (!d_old_pi || !d_old_pj || !d_new_ibeg || !d_new_pj || !d_map)))
        return TMPS_ERR_BAD_ARG;
    if (nold == 0) return TMPS_OK;
    k_pair_map<<<grid_for(nold, kBlk), kBlk, 0, (cudaStream_t)stream>>>(nold, d_old_pi, d_old_pj, d_new_ibeg, d_new_pj,
                                                                        d_map);
    note_launches(1);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_carry(int32_t nold, int32_t nnew, const int32_t* d_map, double* d_old, double* d_new, int32_t reverse,
                   void* stream) {
    if (nold < 0 || nnew < 0 || (nold > 0 && (!d_map || !d_old || (nnew > 0 && !d_new)))) return TMPS_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (!reverse && nnew > 0 && cudaMemsetAsync(d_new, 0, sizeof(double) * 3 * (size_t)nnew, st) != cudaSuccess)
        return TMPS_ERR_CUDA;
    if (nold == 0) return TMPS_OK;
    k_carry<<<grid_for(nold, kBlk), kBlk, 0, st>>>(nold, nnew, d_map, d_old, d_new, reverse);
    note_launches(1);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_setup(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_rec* d_box,
                   const tmps_adj_tape* tape, void* work, void* stream) {
    if (!sys_ok(s) || !p || !d_box || !tape || !work || !tape->shear || !tape->mask) return TMPS_ERR_BAD_ARG;
    if (s->n == 0) return TMPS_OK;
    Chain ch{(cudaStream_t)stream};
    Work W = carve(work, s->n, s->npairs);
    if (s->npairs > 0)
        ch.run(k_pairs, blocks_p(s->npairs), kBlk, *s, to_params(*p), 0, (const double*)s->x, (const double*)s->v,
            (const double*)s->w, d_box, tape->shear, tape->mask, W, (const Queue*)nullptr);
    ch.run(k_gather, blocks_a(s->n), kBlk, *s, p->dt, 0, (const double*)nullptr, (const double*)nullptr, tape->f,
        tape->t, (const uint8_t*)tape->mask, W, (const Queue*)nullptr);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_initial(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_tape* tape,
                     const double* d_xbuild, uint64_t* d_disp, void* stream) {
    if (!sys_ok(s) || !p || !tape || !tape->xh || !tape->vh || !tape->wh || !d_xbuild || !d_disp)
        return TMPS_ERR_BAD_ARG;
    if (s->n == 0) return TMPS_OK;
    Chain ch{(cudaStream_t)stream};
    ch.run(k_initial, grid_for(s->n, kBlk), kBlk, *s, p->dt, *tape, (const double*)nullptr,
        (const tmps_adj_rec*)nullptr, (const tmps_adj_rec*)nullptr, d_xbuild, (unsigned long long*)d_disp,
        (Queue*)nullptr, (int64_t)0, 0.0);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_finish(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_servo* sv,
                    const tmps_adj_tape* tape, tmps_adj_rec* d_rec, int64_t step, void* work, void* stream) {
    if (!sys_ok(s) || !p || !sv || !tape || !d_rec || step < 1 || !work || !tape->xh || !tape->shear || !tape->mask ||
        !tape->f || !tape->t)
        return TMPS_ERR_BAD_ARG;
    Chain ch{(cudaStream_t)stream};
    const int rc = rest_of_step(s, p, sv, *tape, d_rec, step, carve(work, s->n, s->npairs), nullptr, ch);
    if (rc != TMPS_OK) return rc;
    if (s->n > 0)
        ch.run(k_remap, grid_for(s->n, kBlk), kBlk, s->n, (const double*)tape->xh, (const tmps_adj_rec*)(d_rec + (step - 1)),
            (const tmps_adj_rec*)(d_rec + step), s->x, (const Queue*)nullptr);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_forward(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_servo* sv,
                     const tmps_adj_tape* tape, int64_t atom_stride, int64_t pair_stride, tmps_adj_rec* d_rec,
                     int64_t first, int64_t last, const double* d_xbuild, double trigger_sq, int64_t* d_queue, void* work,
                     void* stream) {
    if (!sys_ok(s) || !p || !sv || !tape || !d_rec || first < 1 || last < first || !work || !tape->xh || !tape->vh ||
        !tape->wh || !tape->shear || !tape->mask || !tape->f || !tape->t || !d_queue || !d_xbuild || atom_stride < 0 ||
        pair_stride < 0)
        return TMPS_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    Chain ch{st};
    Work W = carve(work, s->n, s->npairs);
    Queue* q = reinterpret_cast<Queue*>(d_queue);
    if (cudaMemsetAsync(q, 0, sizeof(Queue), st) != cudaSuccess) return TMPS_ERR_CUDA;
    const double* xlast = nullptr;
    tmps_adj_tape t = *tape;
    for (int64_t step = first; step <= last; ++step) {
        t = tape_at(*tape, atom_stride, pair_stride, step - first);
        if (s->n > 0)
            ch.run(k_initial, grid_for(s->n, kBlk), kBlk, *s, p->dt, t, xlast,
                (const tmps_adj_rec*)(step > first ? d_rec + (step - 2) : nullptr), (const tmps_adj_rec*)(d_rec + (step - 1)),
                d_xbuild, (unsigned long long*)nullptr, q, step, trigger_sq);
        const int rc = rest_of_step(s, p, sv, t, d_rec, step, W, q, ch);
        if (rc != TMPS_OK) return rc;
        xlast = t.xh;
    }
    if (s->n > 0)
        ch.run(k_remap, grid_for(s->n, kBlk), kBlk, s->n, (const double*)t.xh, (const tmps_adj_rec*)(d_rec + (last - 1)),
            (const tmps_adj_rec*)(d_rec + last), s->x, (const Queue*)q);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_reverse(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_servo* sv,
                     const tmps_adj_tape* tape, int64_t atom_stride, int64_t pair_stride, const tmps_adj_rec* d_rec,
                     int64_t first, int64_t last, const double* d_fprev, const double* d_tprev, const double* d_xprev,
                     int32_t linked, const double* qbar, const tmps_adj_bar* b, void* work, void* stream) {
    if (!sys_ok(s) || !p || !sv || !tape || !d_rec || first < 1 || last < first || !d_fprev || !d_tprev || !qbar || !b ||
        !work || atom_stride < 0 || pair_stride < 0)
        return TMPS_ERR_BAD_ARG;
    if (!b->x || !b->v || !b->w || !b->f || !b->t || !b->radius || !b->mass || !b->params || !b->box ||
        (s->npairs > 0 && !b->shear))
        return TMPS_ERR_BAD_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    Chain ch{st};
    Work W = carve(work, s->n, s->npairs);
    const int nbA = grid_for(s->n, kBlk), nbP = grid_for(s->npairs, kPairTile);
    if (s->n == 0 && cudaMemsetAsync(W.partk, 0, sizeof(double) * 6 * nbA, st) != cudaSuccess) return TMPS_ERR_CUDA;
    auto rec = [&](int64_t k) { return d_rec + k; };
    const double* none = nullptr;
    for (int64_t step = last; step >= first; --step) {
        const tmps_adj_tape t = tape_at(*tape, atom_stride, pair_stride, step - first);
        if (step == last && !linked) {
            // the remap and the servo of the last step; else the call for the steps after it did them
            if (s->n > 0)
                ch.run(k_b_atoms, nbA, kBlk, *s, p->dt, 0, 0, (const uint8_t*)nullptr, none, none, (const double*)t.xh,
                    rec(step - 1), rec(step), *b, W);
            ch.run(k_b_servo, 1, kOne, *sv, p->dt, step, rec(step - 1), rec(step), qbar[step - first + 1], nbA, nbP, 0, 1, 0,
                *b, W);
        }
        const double* xh = step > first ? tape_at(*tape, atom_stride, pair_stride, step - 1 - first).xh : d_xprev;
        if (s->n > 0) {
            ch.run(k_b_final, nbA, kBlk, *s, p->dt, t, *b, W);
            if (s->npairs > 0)
                ch.run_b_pairs(nbP, *s, to_params(*p), 1, (const double*)t.xh, (const double*)t.vh,
                    (const double*)t.wh, (const double*)t.shear, (const uint8_t*)t.mask, rec(step - 1),
                    (const double*)W.wbar, *b, W);
            const tmps_adj_tape tp = step > first ? tape_at(*tape, atom_stride, pair_stride, step - 1 - first) : t;
            // (with no pairs it follows k_b_final, whose velocities it reads before its wait)
            if (s->npairs == 0) ch.join();
            ch.run(k_b_atoms, nbA, kBlk, *s, p->dt, 1, 1, (const uint8_t*)t.mask,
                step > first ? (const double*)tp.f : d_fprev, step > first ? (const double*)tp.t : d_tprev, xh,
                xh ? rec(step - 2) : rec(step - 1), xh ? rec(step - 1) : rec(step), *b, W);
        }
        // (the slot of record step - 1 takes the image terms of this step's contacts; with no atoms the
        // launch before is another of itself, whose sums it reads before its wait)
        if (s->n == 0) ch.join();
        ch.run(k_b_servo, 1, kOne, *sv, p->dt, step - 1, rec(step > 1 ? step - 2 : 0), rec(step - 1), qbar[step - first], nbA,
            nbP, s->npairs > 0 ? 1 : 0, xh ? 1 : 0, (int)((step - 1) & 1), *b, W);
    }
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

int tmps_adj_step_back(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_servo* sv,
                       const tmps_adj_tape* tape, const tmps_adj_rec* d_rec, int64_t step, const double* d_fprev,
                       const double* d_tprev, double qbar, const tmps_adj_bar* b, void* work, void* stream) {
    const double q[2] = {0.0, qbar};
    return tmps_adj_reverse(s, p, sv, tape, 0, 0, d_rec, step, step, d_fprev, d_tprev, nullptr, 0, q, b, work, stream);
}

int tmps_adj_setup_back(const tmps_adj_sys* s, const tmps_adj_params* p, const tmps_adj_rec* d_box,
                        const tmps_adj_tape* tape, const tmps_adj_bar* b, void* work, void* stream) {
    if (!sys_ok(s) || !p || !d_box || !tape || !b || !work || !b->x || !b->v || !b->w || !b->f || !b->t ||
        !b->radius || !b->mass || !b->params || !b->box || (s->npairs > 0 && (!b->shear || !tape->shear || !tape->mask)))
        return TMPS_ERR_BAD_ARG;
    if (s->n == 0 || s->npairs == 0) return TMPS_OK;
    Chain ch{(cudaStream_t)stream};
    Work W = carve(work, s->n, s->npairs);
    const int nbA = grid_for(s->n, kBlk), nbP = grid_for(s->npairs, kPairTile);
    const double* none = nullptr;
    ch.run_b_pairs(nbP, *s, to_params(*p), 0, (const double*)s->x, (const double*)s->v, (const double*)s->w,
        (const double*)tape->shear, (const uint8_t*)tape->mask, d_box, none, *b, W);
    ch.run(k_b_atoms, nbA, kBlk, *s, p->dt, 1, 0, (const uint8_t*)tape->mask, none, none, none, d_box, d_box, *b, W);
    ch.run(k_b_servo, 1, kOne, tmps_adj_servo{}, p->dt, (int64_t)1, d_box, d_box, 0.0, nbA, nbP, 1, 0, 0, *b, W);
    return ok() ? TMPS_OK : TMPS_ERR_CUDA;
}

}  // extern "C"
