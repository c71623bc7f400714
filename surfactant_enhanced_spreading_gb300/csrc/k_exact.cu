// Kernels whose FP64 arithmetic must round exactly like the reference's:
// cell assignment (the discrete ibox2 / ibox64 / isCentral decisions), the
// intramolecular-correction lists, and the SHAKE / RATTLE velocity-Verlet
// halves with the Nose-Hoover friction.  This translation unit is compiled
// with -fmad=false so no multiply-add is contracted, as in the reference.
#include "k_launch.cuh"

namespace sesp {

static __constant__ Tables cT;

void upload_tables_exact(const Tables &t, cudaStream_t st) {
    cudaMemcpyToSymbolAsync(cT, &t, sizeof(Tables), 0, cudaMemcpyHostToDevice, st);
}

constexpr double IRS = 1.0 / RS;

// (int)(q / s) rounded as the reference divides, from q * (1 / s): with
// |q / s| below 1e6 the product and the rounded quotient differ by less
// than 1e-9, so they truncate alike unless the product lies within 1e-9 of
// an integer, where the division itself decides
__device__ inline int trunc_div(double q, double s, double inv_s) {
    const double t = q * inv_s;
    if (fabs(t - rint(t)) > 1e-9) return (int)t;
    return (int)(q / s);
}
// ibox2 - 1 along one axis, src/ibox.f90:127-139
__device__ inline int rank_axis(const Rep &r, int a, double v) {
    int k = trunc_div((v + r.rhs[a]) * r.nr[a], r.rsd[a], r.irsd[a]);
    return k < 0 ? 0 : (k >= r.nr[a] ? r.nr[a] - 1 : k);
}
// rcen2xtmp, src/init_box_dimensions.f90:40-42, tabulated at upload per
// replica, axis and rank (rsd (rk + 1) / nr - rhs - rsd / nr / 2)
__device__ inline double rcen2_axis(const Dev &d, const Rep &r, int a, int rk) {
    const double *t = d.rcen2 + r.axis0 / 4;
    return t[(a > 0 ? r.nr[0] : 0) + (a > 1 ? r.nr[1] : 0) + rk];
}
// ibox64 along one axis relative to a rank centre, src/ibox.f90:172-186
__device__ inline int local_axis(double v, double c2) {
    int k = trunc_div(v - c2 + 2.0 * RS, RS, IRS);
    return k < 0 ? 0 : (k > 3 ? 3 : k);
}
// global key-cell coordinate along one axis (rank by ibox2, cell by ibox64)
__device__ inline int key_axis(const Dev &d, const Rep &r, int a, double v, int *rk) {
    *rk = rank_axis(r, a, v);
    return 4 * (*rk) + local_axis(v, rcen2_axis(d, r, a, *rk));
}
// isCentral along one axis (src/ibox.f90:101-124): the cell whose
// [centre - rs/2, centre + rs/2) holds v, -1 if none (the product only
// picks the three candidates; the comparisons decide)
__device__ inline int central_axis(const double *cen, int n, double v, double rhs) {
    int k0 = (int)floor((v + rhs) * IRS);
    const double rs2 = RS / 2.0;
    for (int k = k0 - 1; k <= k0 + 1; k++) {
        if (k < 0 || k >= n) continue;
        double c = cen[k];
        if (v < c + rs2 && v >= c - rs2) return k;
    }
    return -1;
}

// the cell a site is Central in, or -1
__device__ inline int central_cell(const Dev &d, const Rep &r, int g) {
    const double *cx = d.axis + r.axis0;
    const double *cy = cx + r.nc[0];
    const double *cz = cy + r.nc[1];
    int ix = central_axis(cx, r.nc[0], d.x[g], r.rhs[0]);
    int iy = central_axis(cy, r.nc[1], d.y[g], r.rhs[1]);
    int iz = central_axis(cz, r.nc[2], d.z[g], r.rhs[2]);
    return (ix < 0 || iy < 0 || iz < 0) ? -1 : cell_index(r, ix, iy, iz);
}

// the packed multipoles cleared for the coming far-field build (all threads of the launch)
__device__ inline void clear_packed(const Dev &d) {
    uint4 *p = (uint4 *)d.pk4;
    for (size_t k = blockIdx.x * blockDim.x + threadIdx.x; k < d.pk_bytes / 16; k += (size_t)gridDim.x * blockDim.x)
        p[k] = make_uint4(0u, 0u, 0u, 0u);
}

// Re-key molecules (src/read_config.f90:44-175 and the delete/add pairs
// src/delete_w1.f90:54-195, src/delete_s.f90:33-43; key site O for water,
// 14 for surfactants) and locate every site in the cell it is Central in.
// A w1 water (all three sites in one rank and one ibox64 cell) has its
// sites located in its key cell, as the reference stores it there.
// Threads [0, nmol) take one molecule each (a water with its sites);
// threads [nmol, nmol + nss) one surfactant site each.
__global__ void k_locate(Dev d, int nmol, const int *smols, int nss) {
    clear_packed(d);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nmol) {
        if (t - nmol >= nss) return;
        const int m = smols[(t - nmol) / NSURF], g = d.mfirst[m] + (t - nmol) % NSURF;
        const int loc = central_cell(d, d.rep[d.mrep[m]], g);
        d.sloc[g] = loc;
        if (loc >= 0) atomicAdd(&d.ccount[loc], 1);
        else atomicAdd(&d.counters[2], 1ull);
        return;
    }
    const int m = t;
    const Rep r = d.rep[d.mrep[m]];
    int g0 = d.mfirst[m];
    int kind = d.mkind[m];
    int ks = kind == 0 ? g0 : g0 + 13;
    double p[3] = {d.x[ks], d.y[ks], d.z[ks]};
    int rk[3], kc[3];
    for (int a = 0; a < 3; a++) kc[a] = key_axis(d, r, a, p[a], &rk[a]);
    int key = cell_index(r, kc[0], kc[1], kc[2]);
    d.mkey[m] = key;
    if (kind != 0) {
        d.mw1[m] = 0;
        return;
    }
    int w1 = 1;
    for (int s = 1; s < 3; s++) {
        double q[3] = {d.x[g0 + s], d.y[g0 + s], d.z[g0 + s]};
        for (int a = 0; a < 3; a++) {
            if (rank_axis(r, a, q[a]) != rk[a]) w1 = 0;
            else if (4 * rk[a] + local_axis(q[a], rcen2_axis(d, r, a, rk[a])) != kc[a]) w1 = 0;
        }
    }
    d.mw1[m] = w1;
    for (int s = 0; s < 3; s++) {
        const int g = g0 + s;
        const int loc = w1 ? key : central_cell(d, r, g);
        d.sloc[g] = loc;
        if (loc >= 0) atomicAdd(&d.ccount[loc], 1);
        else atomicAdd(&d.counters[2], 1ull);
    }
}

// Sites of each surfactant that lie outside the 27-cell block of a site's
// own cell (src/buildinternal.f90:13-63); cells on the 10^3 grid of the
// key rank (ibox1000, rcen1000: src/ibox.f90:206-220,
// src/init_box_dimensions.f90:155-170).  One thread per surfactant site.
__global__ void k_isub(Dev d, int nsurf_sites, const int *surf_mol_of) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsurf_sites) return;
    int m = surf_mol_of[t / NSURF];
    int j = t % NSURF;
    const Rep r = d.rep[d.mrep[m]];
    int g0 = d.mfirst[m];
    int key = d.mkey[m] - r.cell0;
    int kc[3] = {key % r.nc[0], (key / r.nc[0]) % r.nc[1], key / (r.nc[0] * r.nc[1])};
    double pm[3] = {d.x[g0 + j], d.y[g0 + j], d.z[g0 + j]};
    double cen[3];
    for (int a = 0; a < 3; a++) {
        double c2 = rcen2_axis(d, r, a, kc[a] / 4);
        int li = trunc_div(pm[a] - c2 + 5.0 * RS, RS, IRS) + 1;
        cen[a] = 10.0 * RS * li / 10.0 - 10.0 * RS / 2.0 - 10.0 * RS / 20.0 + c2;
    }
    const double r15 = 1.5 * RS;
    uint32_t mask = 0;
    for (int k = 0; k < NSURF; k++) {
        if (k == j) continue;
        double pk[3] = {d.x[g0 + k], d.y[g0 + k], d.z[g0 + k]};
        bool near = true;
        for (int a = 0; a < 3; a++) near = near && (pk[a] < cen[a] + r15 && pk[a] >= cen[a] - r15);
        if (!near) mask |= (1u << k);
    }
    d.isub[t] = mask;
}

// ---------------------------------------------------------------- integrator

// The waters' halves of the plain path.  What bounds them is FP64 issue: a warp
// instruction takes its scheduler's FP64 unit 64 cycles, whatever its active
// lanes, so a water's sweeps take 64 cycles x its warp's instructions.  CTAs
// are single warps, spread over all schedulers; the reciprocal masses, the
// fixed bond vectors and divisions by constants leave the sweeps; and up to
// MOVE_SPLIT_MAX waters, the number that fills every scheduler once, a water
// takes three lanes, one per component (26 FP64 instructions a corrected SHAKE
// bond, 46 with a lane per water; more waters than that are bound by the sum
// over all of them, which a lane per water keeps smaller).  1,000 waters at
// tolerance 1e-8: SHAKE 204 -> 109 us, RATTLE 218 -> 98 us (187 with the
// division of infinities inlined); 20,000 waters (a lane each) 381 -> 254 and
// 417 -> 244 us (346).
constexpr int WATERS_SPLIT = 10;                       // waters of a warp with three lanes each
constexpr int MOVE_SPLIT_MAX = WATERS_SPLIT * 4 * GB300_SMS;
constexpr int MOVE_BLOCK = 32;

// a rare division as a call: inlined, the compiler runs it beside the common
// path for every operand and selects
__device__ __noinline__ double div_call(double a, double b) { return a / b; }

// a / b, correctly rounded, from y = 1 / b correctly rounded (P. Markstein,
// IBM J. Res. Dev. 34, 111 (1990)): the first step brings the quotient within
// an ulp, the second rounds it.  Infinities and NaN take the division.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    q = fma(fma(-q, b, a), y, q);
    if ((__double2hiint(q) & 0x7ff00000) == 0x7ff00000) q = div_call(a, b);
    return q;
}

// a / DT: RN(1 / DT) lies within 0.14 x 2^-53 of 1 / DT, so a y is within an
// ulp of the quotient and the second step alone rounds it
__device__ __forceinline__ double div_dt(double a) {
    constexpr double y = 1.0 / DT;
    double q = a * y;
    q = fma(fma(-q, DT, a), y, q);
    if ((__double2hiint(q) & 0x7ff00000) == 0x7ff00000) q = div_call(a, DT);
    return q;
}

// The plain path's surfactants: the Gauss-Seidel sweeps over 28 bonds of
// src/move_surfactant_a.f90:36-134 and src/move_surfactant_b.f90:30-118, bit
// for bit, as a wavefront of one molecule per warp.  A bond has a fixed step
// within its sweep (SURF_TAU), sweeps follow each other 4 steps apart, and of
// two bonds that share a site the later in the reference's order comes 1 to 3
// steps after the other: each site sees the sequential order's updates.  Six
// sweeps are in flight, seven bonds a step, three lanes each (one per
// component): lane 3 u + a has the main line of sweep u (mod 6), bonds 0..22
// and 27, for u < 6, and the second branch of site 17, bonds 23..26, for u =
// 6.  Once a sweep has changed nothing, neither have the later ones under
// way.  A sum over components is formed by every lane in the reference's
// order from its neighbours' products.
// Bound by FP64 issue and latency along one molecule's steps (a step of a
// correcting bond is 32 FP64 warp instructions; a thread per molecule took 52,
// in sequence over all sweeps, and spilled): 12 surfactants with 701 waters,
// SHAKE 280 -> 60 us, RATTLE 571 -> 58 us (75 and 149 with sweeps 8 apart and
// the division of infinities inlined; the waters bound them now).
struct SurfShared {
    double p[NSURF][3], v[NSURF][3], r[NBOND][3], ke[NSURF];
    double m[NSURF], rm[NSURF], c0[NBOND], c1[NBOND], c2[NBOND];   // masses and their reciprocals; per-bond constants
    int i[NBOND], j[NBOND];
};

// sum of a group's three components (lanes first..first + 2) in the reference's order
__device__ __forceinline__ double sum3(double v, int first) {
    const double a = __shfl_sync(0xffffffffu, v, first), b = __shfl_sync(0xffffffffu, v, first + 1),
                 c = __shfl_sync(0xffffffffu, v, first + 2);
    return a + b + c;
}

// Runs a molecule's sweeps; act(b, on) takes bond b for the lane's group
// (every lane calls it; `on`: the group has a bond in this step) and says
// whether it corrected it.  True if the tolerance was met within maxit + 1
// sweeps.
constexpr int SURF_LAG = 4, SURF_END = 23, SURF_LINES = 6;
template <typename F>
__device__ __forceinline__ bool surf_sweeps(int u, int maxit, F act) {
    if (maxit < 0) return false;
    const bool line = u < SURF_LINES, branch = u == SURF_LINES;
    int sweep = line ? u : 0;
    bool dirty = false, branch_dirty = false;   // in the lane's sweep; on its second branch (kept one step)
    for (int step = 0;; step++) {
        const int tau = step - SURF_LAG * sweep;
        const bool on = sweep <= maxit && (line ? tau >= 0 : branch && tau >= 19 && tau <= 22);
        const int b = on ? (branch ? tau + 4 : tau == SURF_END ? NBOND - 1 : tau) : 0;
        if (act(b, on)) dirty = true;
        const bool ends = line && on && tau == SURF_END;
        const bool bd = __any_sync(0xffffffffu, branch && branch_dirty);
        const unsigned clean = __ballot_sync(0xffffffffu, ends && !dirty && !bd);
        const unsigned out = __ballot_sync(0xffffffffu, ends && sweep == maxit);
        if (ends) { dirty = false; sweep += SURF_LINES; }
        if (branch && tau == 22) { branch_dirty = dirty; dirty = false; sweep++; }
        __syncwarp();
        if (clean) return true;
        if (out) return false;
    }
}

// which group and component a lane has
struct SurfLane {
    int lane, u, a, first;
    __device__ SurfLane() {
        lane = threadIdx.x & 31;
        u = lane / 3; a = lane % 3;
        first = min(lane - a, 29);
    }
};

__device__ void surf_move_a(const Dev &d, const int *mols, double tol, int maxit, SurfShared &s, int block) {
    const SurfLane L;
    for (int k = L.lane; k < NSURF; k += 32) { s.m[k] = cT.mass[2 + k]; s.rm[k] = 1.0 / cT.mass[2 + k]; }
    for (int b = L.lane; b < NBOND; b += 32) {
        const int i = cT.bi[b], j = cT.bj[b];
        s.i[b] = i; s.j[b] = j;
        s.c0[b] = cT.dsqs[b];
        s.c1[b] = cT.dsqs[b] * (2.0 * tol);
        s.c2[b] = 2.0 * (1.0 / cT.mass[2 + i] + 1.0 / cT.mass[2 + j]);
    }
    const int m = mols[block], g0 = d.mfirst[m];
    const double escale = 1.0 - d.eta[d.mrep[m]] * DT / 2.0;
    double *const xs[3] = {d.x, d.y, d.z}, *const vs[3] = {d.vx, d.vy, d.vz}, *const as[3] = {d.ax, d.ay, d.az};
    auto each = [&](auto f) {   // every (site, component)
        for (int k = L.lane; k < 3 * NSURF; k += 32) f(k / 3, k % 3);
        __syncwarp();
    };
    auto kinetic = [&]() {   // sum of m v^2 in site order
        for (int k = L.lane; k < NSURF; k += 32) {
            const double vx = s.v[k][0], vy = s.v[k][1], vz = s.v[k][2];
            s.ke[k] = s.m[k] * (vx * vx + vy * vy + vz * vz);
        }
        __syncwarp();
        double sum = 0.0;
        if (L.lane == 0)
            for (int k = 0; k < NSURF; k++) sum += s.ke[k];
        __syncwarp();
        return sum;
    };
    each([&](int k, int a) { s.p[k][a] = xs[a][g0 + k]; s.v[k][a] = vs[a][g0 + k]; });
    const double ke0 = kinetic();
    for (int k = L.lane; k < 3 * NBOND; k += 32) {
        const int b = k / 3, a = k % 3;
        s.r[b][a] = s.p[s.i[b]][a] - s.p[s.j[b]][a];
    }
    __syncwarp();
    each([&](int k, int a) {
        const double v = s.v[k][a], acc = as[a][g0 + k];
        s.p[k][a] = s.p[k][a] + v * escale + acc;
        s.v[k][a] = v * escale + acc;
    });
    const bool ok = surf_sweeps(L.u, maxit, [&](int b, bool on) {
        const int i = s.i[b], j = s.j[b], a = L.a;
        const double p = s.p[i][a] - s.p[j][a];
        const double diffsq = s.c0[b] - sum3(p * p, L.first);
        const bool cor = on && fabs(diffsq) > s.c1[b];
        if (__any_sync(0xffffffffu, cor)) {
            const double r = s.r[b][a], rpab = sum3(r * p, L.first);
            const double gab = diffsq / (s.c2[b] * rpab);
            if (cor) {
                const double dx = r * gab, di = s.rm[i] * dx, dj = s.rm[j] * dx;
                s.p[i][a] = s.p[i][a] + di; s.p[j][a] = s.p[j][a] - dj;
                s.v[i][a] = s.v[i][a] + di; s.v[j][a] = s.v[j][a] - dj;
            }
        }
        return cor;
    });
    each([&](int k, int a) { xs[a][g0 + k] = s.p[k][a]; vs[a][g0 + k] = s.v[k][a]; });
    const double ke1 = kinetic();
    if (L.lane == 0) {
        d.ke[2 * m] = ke0;
        d.ke[2 * m + 1] = ke1;
        if (!ok) { d.mfail[m] += 1; atomicAdd(&d.counters[0], 1ull); }
    }
}

__device__ void surf_move_b(const Dev &d, const int *mols, double tol, int maxit, SurfShared &s, int block) {
    const SurfLane L;
    for (int k = L.lane; k < NSURF; k += 32) { s.m[k] = cT.mass[2 + k]; s.rm[k] = 1.0 / cT.mass[2 + k]; }
    for (int b = L.lane; b < NBOND; b += 32) {
        const int i = cT.bi[b], j = cT.bj[b];
        s.i[b] = i; s.j[b] = j;
        s.c0[b] = (1.0 / cT.mass[2 + i] + 1.0 / cT.mass[2 + j]) * cT.dsqs[b];
        s.c1[b] = 1.0 / s.c0[b];
    }
    const int m = mols[block], g0 = d.mfirst[m];
    const double escale = 2.0 / (2.0 + d.eta[d.mrep[m]] * DT);
    double *const xs[3] = {d.x, d.y, d.z}, *const vs[3] = {d.vx, d.vy, d.vz}, *const as[3] = {d.ax, d.ay, d.az};
    double *const fs[3] = {d.fx, d.fy, d.fz};
    __syncwarp();   // the constants are in place
    for (int k = L.lane; k < 3 * NSURF; k += 32) {
        const int n = k / 3, a = k % 3;
        const double acc = div_by(fs[a][g0 + n] * DTSQ2, s.m[n], s.rm[n]);
        as[a][g0 + n] = acc;
        s.p[n][a] = xs[a][g0 + n];
        s.v[n][a] = escale * (vs[a][g0 + n] + acc);
    }
    __syncwarp();
    for (int k = L.lane; k < 3 * NBOND; k += 32) {
        const int b = k / 3, a = k % 3;
        s.r[b][a] = s.p[s.i[b]][a] - s.p[s.j[b]][a];
    }
    __syncwarp();
    const bool ok = surf_sweeps(L.u, maxit, [&](int b, bool on) {
        const int i = s.i[b], j = s.j[b], a = L.a;
        const double r = s.r[b][a], v = s.v[i][a] - s.v[j][a];
        const double rvab = div_dt(sum3(r * v, L.first));
        const double gab = div_by(-rvab, s.c0[b], s.c1[b]);
        const bool cor = on && fabs(gab) > tol;
        if (cor) {
            const double dx = r * gab;
            s.v[i][a] = s.v[i][a] + s.rm[i] * dx * DT;
            s.v[j][a] = s.v[j][a] - s.rm[j] * dx * DT;
        }
        return cor;
    });
    for (int k = L.lane; k < 3 * NSURF; k += 32) vs[k % 3][g0 + k / 3] = s.v[k / 3][k % 3];
    if (L.lane == 0 && !ok) { d.mfail[m] += 1; atomicAdd(&d.counters[0], 1ull); }
}

// A water over three lanes, one per component: the same operations in the
// same order as the kernels below (every lane forms the sums over components).
struct WaterLane {
    int a, first;
    bool mine;
    int m, g0;
    __device__ WaterLane(const Dev &d, const int *mols, int nm, int block) {
        const int lane = threadIdx.x & 31, w = block * WATERS_SPLIT + lane / 3;
        a = lane % 3;
        first = min(lane - a, 29);
        mine = lane < 3 * WATERS_SPLIT && w < nm;
        m = mine ? mols[w] : 0;
        g0 = mine ? d.mfirst[m] : 0;
    }
};
__device__ void water_split_a(const Dev &d, const int *mols, int nm, double tol, int maxit, int block) {
    const WaterLane L(d, mols, nm, block);
    double *const x = L.a == 0 ? d.x : L.a == 1 ? d.y : d.z, *const vel = L.a == 0 ? d.vx : L.a == 1 ? d.vy : d.vz;
    const double *const acc = L.a == 0 ? d.ax : L.a == 1 ? d.ay : d.az;
    const double mass[3] = {cT.mass[0], cT.mass[1], cT.mass[1]};
    const double rmO = 1.0 / mass[0], rmH = 1.0 / mass[1], rm[3] = {rmO, rmH, rmH};
    const double escale = L.mine ? 1.0 - d.eta[d.mrep[L.m]] * DT / 2.0 : 1.0;
    double p[3], v[3], r[3], lim[3], mm[3], ke0 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const double vg = L.mine ? vel[L.g0 + i] : 0.0, ag = L.mine ? acc[L.g0 + i] : 0.0;
        ke0 += mass[i] * sum3(vg * vg, L.first);
        p[i] = L.mine ? x[L.g0 + i] : 0.0;
        v[i] = vg * escale + ag;
        r[i] = p[i];
        p[i] = p[i] + vg * escale + ag;
    }
    const double x0 = r[0];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int j = b == 2 ? 0 : b + 1;
        r[b] = r[b] - (b == 2 ? x0 : r[j]);
        lim[b] = cT.dsqw[b] * (2.0 * tol);
        mm[b] = 2.0 * (rm[b] + rm[j]);
    }
    bool ldone = !L.mine;
    for (int it = 0; it <= maxit && __any_sync(0xffffffffu, !ldone); it++) {
        bool clean = true;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int j = b == 2 ? 0 : b + 1;
            const double pab = p[b] - p[j];
            const double diffsq = cT.dsqw[b] - sum3(pab * pab, L.first);
            const bool cor = !ldone && fabs(diffsq) > lim[b];
            if (__any_sync(0xffffffffu, cor)) {
                const double rpab = sum3(r[b] * pab, L.first);
                const double gab = diffsq / (mm[b] * rpab);
                if (cor) {
                    const double dx = r[b] * gab, di = rm[b] * dx, dj = rm[j] * dx;
                    p[b] = p[b] + di; p[j] = p[j] - dj;
                    v[b] = v[b] + di; v[j] = v[j] - dj;
                    clean = false;
                }
            }
        }
        ldone = ldone || clean;
    }
    double ke1 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if (L.mine) { x[L.g0 + i] = p[i]; vel[L.g0 + i] = v[i]; }
        ke1 += mass[i] * sum3(v[i] * v[i], L.first);
    }
    if (L.mine && L.a == 0) {
        d.ke[2 * L.m] = ke0;
        d.ke[2 * L.m + 1] = ke1;
        if (!ldone) { d.mfail[L.m] += 1; atomicAdd(&d.counters[0], 1ull); }
    }
}
__device__ void water_split_b(const Dev &d, const int *mols, int nm, double tol, int maxit, int block) {
    const WaterLane L(d, mols, nm, block);
    const double *const x = L.a == 0 ? d.x : L.a == 1 ? d.y : d.z, *const f = L.a == 0 ? d.fx : L.a == 1 ? d.fy : d.fz;
    double *const vel = L.a == 0 ? d.vx : L.a == 1 ? d.vy : d.vz, *const acc = L.a == 0 ? d.ax : L.a == 1 ? d.ay : d.az;
    const double mass[3] = {cT.mass[0], cT.mass[1], cT.mass[1]};
    const double rmO = 1.0 / mass[0], rmH = 1.0 / mass[1], rm[3] = {rmO, rmH, rmH};
    const double escale = L.mine ? 2.0 / (2.0 + d.eta[d.mrep[L.m]] * DT) : 1.0;
    double xs[3], v[3], r[3], den[3], iden[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        xs[i] = L.mine ? x[L.g0 + i] : 0.0;
        const double ag = div_by(L.mine ? f[L.g0 + i] * DTSQ2 : 0.0, mass[i], rm[i]);
        if (L.mine) acc[L.g0 + i] = ag;
        v[i] = escale * ((L.mine ? vel[L.g0 + i] : 0.0) + ag);
    }
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int j = b == 2 ? 0 : b + 1;
        r[b] = xs[b] - xs[j];
        den[b] = (rm[b] + rm[j]) * cT.dsqw[b];
        iden[b] = 1.0 / den[b];
    }
    bool ldone = !L.mine;
    for (int it = 0; it <= maxit && __any_sync(0xffffffffu, !ldone); it++) {
        bool clean = true;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int j = b == 2 ? 0 : b + 1;
            const double rvab = div_dt(sum3(r[b] * (v[b] - v[j]), L.first));
            const double gab = div_by(-rvab, den[b], iden[b]);
            if (!ldone && fabs(gab) > tol) {
                const double dx = r[b] * gab;
                v[b] = v[b] + rm[b] * dx * DT;
                v[j] = v[j] - rm[j] * dx * DT;
                clean = false;
            }
        }
        ldone = ldone || clean;
    }
    if (L.mine) {
#pragma unroll
        for (int i = 0; i < 3; i++) vel[L.g0 + i] = v[i];
        if (L.a == 0 && !ldone) { d.mfail[L.m] += 1; atomicAdd(&d.counters[0], 1ull); }
    }
}

// move_*_a of a water: Nose-Hoover scaled predictor, SHAKE
// (src/move_w1_a.f90:36-134), and the kinetic sums before and after
// (src/nh_water1.f90)
// (the first CTAs take the surfactants, smols[0..ns))
__global__ void __launch_bounds__(MOVE_BLOCK) k_move_a(Dev d, const int *mols, int nm, const int *smols, int ns, double tol,
                                                      int maxit) {
    __shared__ SurfShared surf;
    const int sb = ns;
    if ((int)blockIdx.x < sb) {
        surf_move_a(d, smols, tol, maxit, surf, blockIdx.x);
        return;
    }
    if (nm <= MOVE_SPLIT_MAX) {
        water_split_a(d, mols, nm, tol, maxit, blockIdx.x - sb);
        return;
    }
    int t = (blockIdx.x - sb) * blockDim.x + threadIdx.x;
    if (t >= nm) return;
    int m = mols[t];
    int rep = d.mrep[m];
    int g0 = d.mfirst[m];
    double escale = 1.0 - d.eta[rep] * DT / 2.0;
    const double mass[3] = {cT.mass[0], cT.mass[1], cT.mass[1]};
    const double rmO = 1.0 / mass[0], rmH = 1.0 / mass[1], rm[3] = {rmO, rmH, rmH};
    double rx[3], ry[3], rz[3], px[3], py[3], pz[3], vx[3], vy[3], vz[3];
    double ke0 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        int g = g0 + i;
        double vxg = d.vx[g], vyg = d.vy[g], vzg = d.vz[g];
        ke0 += mass[i] * (vxg * vxg + vyg * vyg + vzg * vzg);
        rx[i] = d.x[g]; ry[i] = d.y[g]; rz[i] = d.z[g];
        px[i] = d.x[g] + vxg * escale + d.ax[g];
        py[i] = d.y[g] + vyg * escale + d.ay[g];
        pz[i] = d.z[g] + vzg * escale + d.az[g];
        vx[i] = vxg * escale + d.ax[g];
        vy[i] = vyg * escale + d.ay[g];
        vz[i] = vzg * escale + d.az[g];
    }
    double rxab[3], ryab[3], rzab[3], rabsq[3], lim[3], mm[3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int i = b, j = b == 2 ? 0 : b + 1;
        rxab[b] = rx[i] - rx[j]; ryab[b] = ry[i] - ry[j]; rzab[b] = rz[i] - rz[j];
        rabsq[b] = cT.dsqw[b];
        lim[b] = rabsq[b] * (2.0 * tol);
        mm[b] = 2.0 * (rm[i] + rm[j]);
    }
    int it = 0;
    bool ldone = false;
    while (!ldone && it <= maxit) {
        ldone = true;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int i = b, j = b == 2 ? 0 : b + 1;
            double pxab = px[i] - px[j], pyab = py[i] - py[j], pzab = pz[i] - pz[j];
            double pabsq = pxab * pxab + pyab * pyab + pzab * pzab;
            double diffsq = rabsq[b] - pabsq;
            if (fabs(diffsq) > lim[b]) {
                double rpab = rxab[b] * pxab + ryab[b] * pyab + rzab[b] * pzab;
                double rma = rm[i], rmb = rm[j];
                double gab = diffsq / (mm[b] * rpab);
                double dx = rxab[b] * gab, dy = ryab[b] * gab, dz = rzab[b] * gab;
                px[i] = px[i] + rma * dx; py[i] = py[i] + rma * dy; pz[i] = pz[i] + rma * dz;
                px[j] = px[j] - rmb * dx; py[j] = py[j] - rmb * dy; pz[j] = pz[j] - rmb * dz;
                vx[i] = vx[i] + rma * dx; vy[i] = vy[i] + rma * dy; vz[i] = vz[i] + rma * dz;
                vx[j] = vx[j] - rmb * dx; vy[j] = vy[j] - rmb * dy; vz[j] = vz[j] - rmb * dz;
                ldone = false;
            }
        }
        it++;
    }
    double ke1 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        int g = g0 + i;
        d.x[g] = px[i]; d.y[g] = py[i]; d.z[g] = pz[i];
        d.vx[g] = vx[i]; d.vy[g] = vy[i]; d.vz[g] = vz[i];
        ke1 += mass[i] * (vx[i] * vx[i] + vy[i] * vy[i] + vz[i] * vz[i]);
    }
    d.ke[2 * m] = ke0;
    d.ke[2 * m + 1] = ke1;
    if (!ldone) { d.mfail[m] += 1; atomicAdd(&d.counters[0], 1ull); }
}

// eta update of src/move_w2_a.f90:145-157.  ETA_BLOCKS blocks per replica
// each sum a fixed contiguous share of its molecules' kinetic sums
// (thread-strided, then a tree); the last of them to finish adds the shares
// in block order and updates eta.  The summation order is fixed, whichever
// block finishes last; nothing waits.
constexpr int ETA_BLOCKS = 32, ETA_THREADS = 256;
__global__ void __launch_bounds__(ETA_THREADS) k_eta(Dev d) {
    const int rep = blockIdx.x / ETA_BLOCKS, j = blockIdx.x % ETA_BLOCKS;
    const Rep r = d.rep[rep];
    __shared__ double s0[ETA_THREADS], s1[ETA_THREADS];
    __shared__ bool last;
    const int per = (r.nmol + ETA_BLOCKS - 1) / ETA_BLOCKS;
    const int m0 = r.mol0 + j * per, m1 = min(r.mol0 + r.nmol, m0 + per);
    double a = 0.0, b = 0.0;
    for (int m = m0 + threadIdx.x; m < m1; m += ETA_THREADS) { a += d.ke[2 * m]; b += d.ke[2 * m + 1]; }
    s0[threadIdx.x] = a; s1[threadIdx.x] = b;
    __syncthreads();
    for (int w = ETA_THREADS / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) { s0[threadIdx.x] += s0[threadIdx.x + w]; s1[threadIdx.x] += s1[threadIdx.x + w]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        d.eta_part[2 * blockIdx.x] = s0[0];
        d.eta_part[2 * blockIdx.x + 1] = s1[0];
        __threadfence();
        last = atomicAdd(&d.eta_ctl[rep], 1u) == ETA_BLOCKS - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        const volatile double *p = d.eta_part + 2 * ETA_BLOCKS * rep;
        double sum1 = 0.0, sum2 = 0.0;
        for (int k = 0; k < ETA_BLOCKS; k++) { sum1 += p[2 * k]; sum2 += p[2 * k + 1]; }
        sum1 = sum1 / (DT * DT);
        sum2 = sum2 / (DT * DT);
        d.eta[rep] = d.eta[rep] + r.pnh1 * (sum1 + r.pnh2 + sum2);
        d.eta_ctl[rep] = 0u;
    }
}

// move_*_b of a water: acceleration from force, friction, RATTLE
// (src/move_w1_b.f90:30-119)
// (the first CTAs take the surfactants, smols[0..ns))
__global__ void __launch_bounds__(MOVE_BLOCK) k_move_b(Dev d, const int *mols, int nm, const int *smols, int ns, double tol,
                                                      int maxit) {
    __shared__ SurfShared surf;
    const int sb = ns;
    if ((int)blockIdx.x < sb) {
        surf_move_b(d, smols, tol, maxit, surf, blockIdx.x);
        return;
    }
    if (nm <= MOVE_SPLIT_MAX) {
        water_split_b(d, mols, nm, tol, maxit, blockIdx.x - sb);
        return;
    }
    int t = (blockIdx.x - sb) * blockDim.x + threadIdx.x;
    if (t >= nm) return;
    int m = mols[t];
    int rep = d.mrep[m];
    int g0 = d.mfirst[m];
    double escale = 2.0 / (2.0 + d.eta[rep] * DT);
    const double mass[3] = {cT.mass[0], cT.mass[1], cT.mass[1]};
    const double rmO = 1.0 / mass[0], rmH = 1.0 / mass[1], rm[3] = {rmO, rmH, rmH};
    double rx[3], ry[3], rz[3], vx[3], vy[3], vz[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        int g = g0 + i;
        double mi = mass[i], yi = rm[i];
        rx[i] = d.x[g]; ry[i] = d.y[g]; rz[i] = d.z[g];
        double axg = div_by(d.fx[g] * DTSQ2, mi, yi), ayg = div_by(d.fy[g] * DTSQ2, mi, yi), azg = div_by(d.fz[g] * DTSQ2, mi, yi);
        d.ax[g] = axg; d.ay[g] = ayg; d.az[g] = azg;
        vx[i] = escale * (d.vx[g] + axg);
        vy[i] = escale * (d.vy[g] + ayg);
        vz[i] = escale * (d.vz[g] + azg);
    }
    double rxab[3], ryab[3], rzab[3], den[3], iden[3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int i = b, j = b == 2 ? 0 : b + 1;
        rxab[b] = rx[i] - rx[j]; ryab[b] = ry[i] - ry[j]; rzab[b] = rz[i] - rz[j];
        den[b] = (rm[i] + rm[j]) * cT.dsqw[b];
        iden[b] = 1.0 / den[b];
    }
    int it = 0;
    bool ldone = false;
    while (!ldone && it <= maxit) {
        ldone = true;
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int i = b, j = b == 2 ? 0 : b + 1;
            double vxab = vx[i] - vx[j], vyab = vy[i] - vy[j], vzab = vz[i] - vz[j];
            double rvab = rxab[b] * vxab + ryab[b] * vyab + rzab[b] * vzab;
            double rma = rm[i], rmb = rm[j];
            rvab = div_dt(rvab);
            double gab = div_by(-rvab, den[b], iden[b]);
            if (fabs(gab) > tol) {
                double dx = rxab[b] * gab, dy = ryab[b] * gab, dz = rzab[b] * gab;
                vx[i] = vx[i] + rma * dx * DT; vy[i] = vy[i] + rma * dy * DT; vz[i] = vz[i] + rma * dz * DT;
                vx[j] = vx[j] - rmb * dx * DT; vy[j] = vy[j] - rmb * dy * DT; vz[j] = vz[j] - rmb * dz * DT;
                ldone = false;
            }
        }
        it++;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        int g = g0 + i;
        d.vx[g] = vx[i]; d.vy[g] = vy[i]; d.vz[g] = vz[i];
    }
    if (!ldone) { d.mfail[m] += 1; atomicAdd(&d.counters[0], 1ull); }
}

// src/init_accel.f90:10-46
__global__ void k_init_accel(Dev d, int nsite) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nsite) return;
    double m = d.tmass[d.ptype[g]];
    d.ax[g] = d.fx[g] * DTSQ2 / m;
    d.ay[g] = d.fy[g] * DTSQ2 / m;
    d.az[g] = d.fz[g] * DTSQ2 / m;
}

// ---------------------------------------------------------------- configuration preset

// floor division (b > 0)
__device__ inline int floor_div(int a, int b) { const int q = a / b; return (a % b != 0 && a < 0) ? q - 1 : q; }

// Periodic cell location (configuration preset), one thread per site: the
// cell index along each axis is floor((r + rhs) / rs); x and y are wrapped
// into the box and the integer image is kept (positions stay unwrapped, so
// molecules stay whole); a site outside the z range is in no cell.  The
// molecule's key is the cell of its first site.
__global__ void k_locate_cfg(Dev d, int nsite) {
    clear_packed(d);
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nsite) return;
    const int m = d.smol[g];
    const Rep r = d.rep[d.mrep[m]];
    const double x = d.x[g], y = d.y[g], z = d.z[g];
    int loc = -1, kx = 0, ky = 0;
    const double lim = 1e9;   // far outside any box: treated as lost (no cell)
    if (fabs(x) < lim && fabs(y) < lim && fabs(z) < lim) {
        const int ex = (int)floor((x + r.rhs[0]) * IRS), ey = (int)floor((y + r.rhs[1]) * IRS);
        const int ez = (int)floor((z + r.rhs[2]) * IRS);
        kx = floor_div(ex, r.nc[0]);
        ky = floor_div(ey, r.nc[1]);
        if (ez >= 0 && ez < r.nc[2] && abs(kx) < 30000 && abs(ky) < 30000)
            loc = cell_index(r, ex - kx * r.nc[0], ey - ky * r.nc[1], ez);
    }
    d.sloc[g] = loc;
    d.simg[g] = make_short2((short)(loc >= 0 ? kx : 0), (short)(loc >= 0 ? ky : 0));
    if (loc >= 0) atomicAdd(&d.ccount[loc], 1);
    else atomicAdd(&d.counters[2], 1ull);
    if (g == d.mfirst[m]) { d.mkey[m] = loc; d.mw1[m] = 0; }
}

// Same-molecule sites of each chain bead whose (unwrapped) cells are not
// adjacent to the bead's own: the pairs the far field counts and the
// correction removes.  One thread per bead.
__global__ void k_isub_cfg(Dev d, int nbeads, const int *chain_mols) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nbeads) return;
    const int m = chain_mols[t / NCH], j = t % NCH;
    const Rep r = d.rep[d.mrep[m]];
    const int g0 = d.mfirst[m];
    auto ext = [&](int g, int a) {
        const double v = a == 0 ? d.x[g] : (a == 1 ? d.y[g] : d.z[g]);
        const double c = fabs(v) < 1e9 ? floor((v + r.rhs[a]) * IRS) : 0.0;
        return (int)c;
    };
    const int ej[3] = {ext(g0 + j, 0), ext(g0 + j, 1), ext(g0 + j, 2)};
    uint32_t mask = 0;
    for (int k = 0; k < NCH; k++) {
        if (k == j) continue;
        const int g = g0 + k;
        if (abs(ext(g, 0) - ej[0]) > 1 || abs(ext(g, 1) - ej[1]) > 1 || abs(ext(g, 2) - ej[2]) > 1) mask |= 1u << k;
    }
    d.isub[t] = mask;
}

// move_a of flexible chains: the Nose-Hoover scaled predictor of
// src/move_surfactant_a.f90:36-60 with no constraint, and the kinetic sums
// before and after.  16 lanes per chain, one bead each; the sums are added
// by a fixed shuffle tree within the 16 lanes.
__global__ void k_move_free_a(Dev d, const int *mols, int nm) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int q = t >> 4, i = t & 15;
    double ke0 = 0.0, ke1 = 0.0;
    if (q < nm && i < NCH) {
        const int m = mols[q], g = d.mfirst[m] + i;
        const double escale = 1.0 - d.eta[d.mrep[m]] * DT / 2.0;
        const double mi = d.tmass[d.ptype[g]];
        double vx = d.vx[g], vy = d.vy[g], vz = d.vz[g];
        ke0 = mi * (vx * vx + vy * vy + vz * vz);
        d.x[g] = d.x[g] + vx * escale + d.ax[g];
        d.y[g] = d.y[g] + vy * escale + d.ay[g];
        d.z[g] = d.z[g] + vz * escale + d.az[g];
        vx = vx * escale + d.ax[g]; vy = vy * escale + d.ay[g]; vz = vz * escale + d.az[g];
        d.vx[g] = vx; d.vy[g] = vy; d.vz[g] = vz;
        ke1 = mi * (vx * vx + vy * vy + vz * vz);
    }
    for (int o = 8; o > 0; o >>= 1) {
        ke0 += __shfl_xor_sync(0xffffffffu, ke0, o);
        ke1 += __shfl_xor_sync(0xffffffffu, ke1, o);
    }
    if (q < nm && i == 0) {
        const int m = mols[q];
        d.ke[2 * m] = ke0;
        d.ke[2 * m + 1] = ke1;
    }
}

// move_b of flexible chains: acceleration from force and friction
// (src/move_surfactant_b.f90:30-55) with no constraint
__global__ void k_move_free_b(Dev d, const int *mols, int nm) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nm * NCH) return;
    const int m = mols[t / NCH], g = d.mfirst[m] + t % NCH;
    const double escale = 2.0 / (2.0 + d.eta[d.mrep[m]] * DT);
    const double mi = d.tmass[d.ptype[g]];
    const double axg = d.fx[g] * DTSQ2 / mi, ayg = d.fy[g] * DTSQ2 / mi, azg = d.fz[g] * DTSQ2 / mi;
    d.ax[g] = axg; d.ay[g] = ayg; d.az[g] = azg;
    d.vx[g] = escale * (d.vx[g] + axg);
    d.vy[g] = escale * (d.vy[g] + ayg);
    d.vz[g] = escale * (d.vz[g] + azg);
}

// ---------------------------------------------------------------- launchers

void launch_locate(const Dev &d, int nmol, const int *smols, int nsurf_sites, int per, int nsite, cudaStream_t st) {
    if (per) k_locate_cfg<<<(nsite + 127) / 128, 128, 0, st>>>(d, nsite);
    else k_locate<<<(nmol + nsurf_sites + 127) / 128, 128, 0, st>>>(d, nmol, smols, nsurf_sites);
}
void launch_isub(const Dev &d, int nsurf_sites, const int *surf_mols, int per, cudaStream_t st) {
    if (!nsurf_sites) return;
    if (per) k_isub_cfg<<<(nsurf_sites + 127) / 128, 128, 0, st>>>(d, nsurf_sites, surf_mols);
    else k_isub<<<(nsurf_sites + 31) / 32, 32, 0, st>>>(d, nsurf_sites, surf_mols);
}
static int move_blocks(int nw, int ns) {
    const int w = nw <= MOVE_SPLIT_MAX ? WATERS_SPLIT : MOVE_BLOCK;
    return ns + (nw + w - 1) / w;
}
// fast = 0 (plain path): the FP64 sweeps above, dividing exactly as the
// reference does; fast = 1 / 2 (mixed paths): the FP64 / FP32 sweeps of
// k_constraint.cu.
void launch_move_a(const Dev &d, const int *wmols, int nw, const int *smols, int ns, int nrep, int nmol, int nsite,
                   double tol, int maxit, int fast, const ConstraintShape &sh, int chains, cudaStream_t st) {
    if (chains) {   // flexible chains: constraints on the waters only
        if (fast && fast != 2) {
            launch_move_a_mat(d, nw, smols, ns, nmol, nsite, sh, st, tol, maxit);
            return;
        }
        if (fast) launch_move_a32(d, nw, smols, 0, nmol, nsite, sh, st, tol, maxit, 1);
        else if (nw) k_move_a<<<move_blocks(nw, 0), MOVE_BLOCK, 0, st>>>(d, wmols, nw, smols, 0, tol, maxit);
        if (ns) k_move_free_a<<<(ns * 16 + 127) / 128, 128, 0, st>>>(d, smols, ns);
        return;
    }
    if (fast) {
        launch_move_a32(d, nw, smols, ns, nmol, nsite, sh, st, tol, maxit, fast == 2);
    } else {
        if (nw + ns) k_move_a<<<move_blocks(nw, ns), MOVE_BLOCK, 0, st>>>(d, wmols, nw, smols, ns, tol, maxit);
    }
}
void launch_eta(const Dev &d, int nrep, cudaStream_t st) { k_eta<<<nrep * ETA_BLOCKS, ETA_THREADS, 0, st>>>(d); }
void launch_move_b(const Dev &d, const int *wmols, int nw, const int *smols, int ns, int nmol, int nsite, double tol,
                   int maxit, int fast, const ConstraintShape &sh, int chains, cudaStream_t st) {
    if (chains) {
        if (fast && fast != 2) {
            launch_move_b_mat(d, nw, smols, ns, nmol, nsite, sh, st, tol, maxit);
            return;
        }
        if (fast) launch_move_b32(d, nw, smols, 0, nmol, nsite, sh, st, tol, maxit, 1);
        else if (nw) k_move_b<<<move_blocks(nw, 0), MOVE_BLOCK, 0, st>>>(d, wmols, nw, smols, 0, tol, maxit);
        if (ns) k_move_free_b<<<(ns * NCH + 255) / 256, 256, 0, st>>>(d, smols, ns);
        return;
    }
    if (fast) {
        launch_move_b32(d, nw, smols, ns, nmol, nsite, sh, st, tol, maxit, fast == 2);
    } else {
        if (nw + ns) k_move_b<<<move_blocks(nw, ns), MOVE_BLOCK, 0, st>>>(d, wmols, nw, smols, ns, tol, maxit);
    }
}
void launch_init_accel(const Dev &d, int nsite, cudaStream_t st) {
    k_init_accel<<<(nsite + 255) / 256, 256, 0, st>>>(d, nsite);
}

}  // namespace sesp
