// Physics kernels of the VVM step (everything except the elliptic solves).
//
// T is the storage and stencil arithmetic type: double for the plain FP64
// step, float for the mixed-precision step. Profiles stay double and are
// rounded to T on load. Domain-wide sums always accumulate in double.
//
// Each kernel restates one or more reference routines and keeps their index
// ranges, boundary treatment and expression order; the file:line citations
// name the reference code. Halo fills are fused into the producing kernel
// (store_center / store_westdown write every ghost image of a cell).
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "gs_bands.cuh"
#include "vvm_common.cuh"

namespace vvm {

// Per-level coefficient profiles precomputed on the host (double, [nz]),
// each formed with the reference's own expression.
struct Profiles {
    const double *rhou, *rhow, *thvb, *thb_init, *qvb0, *pib, *pb, *lambda2;
    const double *vt_c1;      // (1E-3*rhow[k])*0.5            Advection.cpp:165
    const double *vt_fac;     // pow(rhow[k]/rhow[1], -0.5)    Advection.cpp:165
    const double *pc;         // 380/(pow(pib,Cp/Rd)*P0)       MicroPhysics.cpp:10,82
    const double *lvcp;       // Lv/(Cp*pib)                    MicroPhysics.cpp:24,108
    const double *dtcgr_th;   // dt*CGR of Nudge_theta (0 below k_start)
    const double *dtcgr_zeta; // dt*CGR of Nudge_zeta (0 below k_start or case 2)
    const double *q1ls, *q2ls;  // large-scale forcing profiles (may be all zero)
    double pf1, pf2;          // 1E-3*rhou[1], pow(rhou[1]/rhow[1], -0.5)  Iteration.cpp:115
    // Mixed step only: th and qv are stored as perturbations from the
    // reference profiles ref[0] = th0 (thb_init) and ref[1] = qv0 (qvb0).
    // For each: d0[k] = ref[k] - ref[k-1], s0[k] = ref[k] + ref[k-1],
    // g0[k] = ref[k+1] - ref[k-1], dn[k] = ref[k] - (nudging target)[k].
    const double *ref[2], *d0[2], *s0[2], *g0[2], *dn[2];
    // Vertical level metric (the reference's constants on uniform levels,
    // exactly; see upload_profiles): flux divergences at centres (r2dzc =
    // 1/(2 dc)) and faces (r2dzw = 1/(2 dw)), the w gradient across a centre
    // (rdzc = 1/dc), gradients across two centres (r2dzcc = 1/(z[k+1]-z[k-1])),
    // the eddy-coefficient cap (kmax = 0.8 dx dc / dt), the Gauss-Seidel
    // vertical factors of Mparam (gsM_*) and Hparam (gsS_*): cz = rdz2_k dt /
    // rho and the down term's density times its spacing ratio, and cal_u's
    // centre-to-centre spacing (dzw) and top factor (hfac = dx / dc_top, 1 on
    // uniform levels as the reference has it); pubarTop's top spacings.
    const double *r2dzc, *r2dzw, *rdzc, *r2dzcc, *kmax, *gsM_cz, *gsM_rhod, *gsS_cz, *gsS_rhod, *dzw;
    double rdz_up, rdz_dn, rdz_c, hfac;
};

// True for the mixed step, whose th and qv arrays hold perturbations.
template <typename T>
constexpr bool kPert = std::is_same<T, float>::value;

// AB2 bookkeeping shared by every prognostic tendency
// (e.g. Advection.cpp:69-71): slot (step+1)%2 receives the new tendency,
// slot step%2 holds the previous one, and on step 0 both become the new one.
struct AB2 {
    int sn, so, first;
    __host__ __device__ static AB2 of(int step) { return AB2{(step + 1) & 1, step & 1, step == 0}; }
};

template <typename T>
__device__ __forceinline__ T ab2_push(T* hn, T* ho, size_t idx, T tend, const AB2& s) {
    T old = s.first ? tend : ho[idx];
    hn[idx] = tend;
    if (s.first) ho[idx] = tend;
    return old;
}

// cp.async helpers: 16-byte global -> shared copies, grouped per row.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// One element global -> shared, asynchronous (cp.async, 4 or 8 bytes).
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem, const T* gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// ---------------------------------------------------------------------------
// Domain-mean top wind tendency (PoissonSolver::pubarTop_pt,
// PoissonSolver.cpp:655-676). One block; in a whole step an extra block of
// k_pzeta, which reads the same time level (a launch of its own stood 9 us at
// the head of the scalars' chain).

template <typename T>
struct PubarArgs {
    Dims d;
    Consts c;
    Profiles p;
    const T *u, *w, *RKM;
    double* ubar;     // [0] ubarTop, [1] ubarTopp
    double* dubar;    // dubarTop_advect[2]
    AB2 ab;
};

template <typename T>
__device__ __forceinline__ void k_pubartop_body(const PubarArgs<T>& a) {
    __shared__ double sh[32 * 3];
    const Dims& d = a.d;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nt = blockDim.x * blockDim.y;
    const int t = d.nz - 2, b = d.nz - 3, top = d.nz - 1;
    const double* rhou = a.p.rhou;
    const double* rhow = a.p.rhow;
    double s[3] = {0, 0, 0};
#pragma unroll 4
    for (int i = 1 + tid; i < d.nx - 1; i += nt) {
        double ut = a.u[d.at(i, t)], ub = a.u[d.at(i, b)], utop = a.u[d.at(i, top)];
        double wt = a.w[d.at(i, t)], wtm = a.w[d.at(i - 1, t)];
        const T* K = a.RKM;
        s[0] += 0.25 * (rhou[t] * ut + rhou[b] * ub) * (wt + wtm);
        s[1] += rhow[top] * 0.25 * ((double)K[d.at(i, top)] + K[d.at(i, t)] + K[d.at(i - 1, top)] + K[d.at(i - 1, t)]) *
                (a.p.rdz_up * (utop - ut));
        s[2] += rhow[t] * 0.25 * ((double)K[d.at(i, t)] + K[d.at(i, b)] + K[d.at(i - 1, t)] + K[d.at(i - 1, b)]) *
                (a.c.rdx * (wt - wtm) + a.p.rdz_dn * (ut - ub));
    }
    block_sum(s, sh);
    if (tid == 0) {
        double n = (double)(d.nx - 2.);
        double down = s[0] / n, kup = s[1] / n, kdown = s[2] / n;
        double pa = (-down) * a.p.rdz_c / rhou[t];
        double pb = (kup - kdown) * a.p.rdz_c / rhou[t];
        double tend = -pa + pb;
        double old = a.ab.first ? tend : a.dubar[a.ab.so];
        a.dubar[a.ab.sn] = tend;
        if (a.ab.first) a.dubar[a.ab.so] = tend;
        a.ubar[1] = a.ubar[0] + 1.5 * a.c.dt * tend - 0.5 * a.c.dt * old;
    }
}
constexpr int kPubarThreads = 1024;   // of k_pubartop, at most
template <typename T>
__global__ void __launch_bounds__(kPubarThreads) k_pubartop(PubarArgs<T> a) { k_pubartop_body<T>(a); }

// ---------------------------------------------------------------------------
// Vorticity advection + buoyancy + westdown halo of zetap
// (Iteration::pzeta_pt: Advection.cpp:84-149, Buoyancy.cpp:11-58,
// Boundary.cpp:21-30). One thread per interior zeta point (i, k),
// i = 1..nx-2, k = 2..nz-2.

template <typename T>
struct PZetaArgs {
    Dims d;
    Consts c;
    Profiles p;
    const T *zeta, *u, *w, *th, *qv, *qc, *qr;
    T* zetap;
    T *hz_n, *hz_o, *hb_n, *hb_o;  // dzeta_advect, dth_buoyancy slots
    int* err;                      // device error word (kStageErrWait), may be null
    AB2 ab;
    PubarArgs<T> pubar;            // pubarTop_pt, by one block past the tiles
    int do_pubar;
    unsigned* kmax;                // [2]: cleared by that block for this step's k_rkm_rkh
    int* redo;                     // and this for its k_gs_sweep
};

// Tile of k_pzeta: 31 x 8R zeta points a block of 32 x 8 threads, R rows a
// thread. zeta, u, w, th, qv, qc and qr are staged by TMA (one box a field).
// A lane is the x face fi = i0 - 1 + lane and the point west of it: it
// evaluates the face once and takes its point's west flux from the lane before
// (lane 0 owns no point). Going up its rows it carries the z flux, the staggered
// mass fluxes Uw, Wu (Advection.cpp:90-91) and the buoyancy difference of the
// row below, so each is formed once. As in k_padv one square root a face, no
// division but the buoyancy's by thvb. Bound by instruction issue: 28 -> 22 us
// at 2048 x 256 FP64, 25 -> 16 FP32; 96 -> 57 and 84 -> 42 at 8192 x 256 (from
// staging loops that divide for their indexes, two roots a face and every flux
// through shared memory).
constexpr int kStageErrWait = 4;   // device error word: a stencil's TMA staging wait gave up
constexpr int kTileLanes = 32, kTileWarps = 8, kTileBX = 31;   // blocks of k_pzeta and k_padv
// The staged box of one field: the tile's rows with two halo rows a side and 40
// columns from the halo's first one, i0-2, rounded down to a 16-byte boundary
// (TMA requires x * element size to be a multiple of 16).
constexpr int kTileVX = 40;
constexpr int tile_rows(int R) { return kTileWarps * R; }

// Tensor maps of a tile kernel's fields (box kTileVX by its staged rows).
template <int N>
struct FieldMaps {
    CUtensorMap m[N];
};

// The velocity part of one face's flux, shared by every advected field:
// flux = base (v0 + vm) - 1/3 (c (v0 - vm) - s dv), dv the difference across
// the upwind neighbour face (Advection.cpp:36-50, :107-118 with the terms that
// the wind's sign makes zero left out); c = s = 0 next to the boundaries.
template <typename T>
struct Face {
    T base, c, s;
    bool pos;   // wind towards +
};
// base: the face's mass flux; mm, mp: the densities times winds vm, vp of the
// neighbour faces on either side enter as mm * vm, mp * vp.
template <typename T>
__device__ __forceinline__ Face<T> face_of(bool hi, T base, T mm, T vm, T mp, T vp) {
    Face<T> F;
    F.base = base;
    F.pos = base > T(0);
    F.c = F.s = T(0);
    if (hi) {
        F.c = fabs(base);
        F.s = sqrt(fabs(base * (F.pos ? mm : mp) * (F.pos ? plus_part(vm) : minus_part(vp))));
    }
    return F;
}
template <typename T>
__device__ __forceinline__ T face_flux(const Face<T>& F, T d, T dm, T dp, T sum) {
    return F.base * sum + T(-1. / 3.) * (F.c * d - F.s * (F.pos ? dm : dp));
}

template <typename T, int R>
struct PZetaShared {
    static constexpr int BZ = tile_rows(R), VZ = BZ + 4;
    T v[7][VZ][kTileVX];     // zeta, u, w, th, qv, qc, qr: rows k0-2..
    // rows k0-2 .. k0+BZ+2: rhou, rhow, r2dx / rhow, r2dzw / rhow, g / rhow,
    // thvb; mixed: the reference th0, qv0
    T row[BZ + 5][kPert<T> ? 8 : 6];
};

template <typename T, int R>
__device__ __forceinline__ void k_pzeta_body(const FieldMaps<7>& maps, const PZetaArgs<T>& a) {
    using Sh = PZetaShared<T, R>;
    constexpr int BZ = Sh::BZ, VZ = Sh::VZ, VX = kTileVX, AL = 16 / sizeof(T);
    if (a.do_pubar && blockIdx.y == 0) {   // the first row of blocks: it starts with the first wave
        if (blockIdx.x == 0) {
            if (threadIdx.x == 0 && threadIdx.y == 0) {
                a.kmax[0] = a.kmax[1] = 0u;
                *a.redo = 0;
            }
            k_pubartop_body<T>(a.pubar);
        }
        return;
    }
    const int by = blockIdx.y - (a.do_pubar ? 1 : 0);
    extern __shared__ __align__(128) unsigned char pzeta_smem[];
    __shared__ uint64_t stage_bar;
    Sh& S = *reinterpret_cast<Sh*>(pzeta_smem);
    const Dims& d = a.d;
    const int lane = threadIdx.x, wid = threadIdx.y, tid = lane + kTileLanes * wid;
    const int i0 = 1 + blockIdx.x * kTileBX, k0 = 2 + by * BZ;
    const int x0 = (i0 - 2) & ~(AL - 1);
    const int i = i0 - 1 + lane;   // the lane's face, and the point west of it

    const uint32_t bar = smem_u32(&stage_bar);
    if (tid == 0) mbar_init1(bar);
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(bar, 7 * VZ * VX * sizeof(T));
#pragma unroll
        for (int f = 0; f < 7; f++) tma_load_2d(smem_u32(&S.v[f][0][0]), &maps.m[f], x0, k0 - 2, bar);
    }
    for (int t = tid; t < BZ + 5; t += kTileLanes * kTileWarps) {
        const int k = k0 - 2 + t;
        if (k > d.nz - 1) break;
        T* r = S.row[t];
        r[0] = T(a.p.rhou[k]);
        r[1] = T(a.p.rhow[k]);
        r[2] = T(a.c.r2dx) / r[1];
        r[3] = T(a.p.r2dzw[k]) / r[1];
        r[4] = T(a.c.gravity) / r[1];
        r[5] = T(a.p.thvb[k]);
        if constexpr (kPert<T>) {
            r[6] = T(a.p.ref[0][k]);
            r[7] = T(a.p.ref[1][k]);
        }
    }
    const bool ok = mbar_wait_bounded(bar, 0);
    if (__syncthreads_or(!ok)) {   // the copies never landed: report and leave
        if (tid == 0 && a.err) atomicOr(a.err, kStageErrWait);
        mbar_wait_bounded(bar, 0);
        return;
    }

    const int c = i - x0;
    const bool point = lane >= 1 && i <= d.nx - 2;
    const bool wrap = (i == 0);    // the west face of point 1: the halo copy of face nx-2 (Advection.cpp:123)
    const bool xhi = i >= 2 && i <= d.nx - 3;
    const T dt15 = T(1.5 * a.c.dt), dt05 = T(0.5 * a.c.dt);
    const T* const zeta = &S.v[0][0][c];
    const T* const u = &S.v[1][0][c];
    const T* const w = &S.v[2][0][c];
    auto row = [&](int k) { return S.row[k - k0 + 2]; };
    auto at = [&](int k) { return (k - k0 + 2) * VX; };
    auto su = [&](int k, int e) { return row(k)[0] * (u[at(k) + e + 1] + u[at(k) + e]); };    // rhou (u_{i+1} + u_i) at i + e
    auto sw = [&](int k) { return row(k)[1] * (w[at(k)] + w[at(k) - 1]); };                  // rhow (w_i + w_{i-1})
    // flux_w at face k (between rows k and k+1) from Wu there and beside it
    auto zflux = [&](int k, T Wm, T W, T Wp) {
        const T* z = zeta + at(k);
        const Face<T> F = face_of(xhi && k >= 2 && k <= d.nz - 3, W, T(1), Wm, T(1), Wp);
        return face_flux(F, z[VX] - z[0], z[0] - z[-VX], z[2 * VX] - z[VX], z[VX] + z[0]);
    };
    // (thv_i - thv_{i-1}) / thvb of row k (Buoyancy.cpp:3-9, :25-28)
    auto thv_dx = [&](int k) {
        const T *th = &S.v[3][0][c] + at(k), *qv = &S.v[4][0][c] + at(k), *r = row(k);
        if constexpr (!kPert<T>) {
            return (th[0] * (T(1) + T(0.608) * qv[0]) - th[-1] * (T(1) + T(0.608) * qv[-1])) / r[5];
        } else {
            // from perturbations th', qv' about th0(k), qv0(k): dth' + 0.608
            // (th0 dqv' + qv0 dth' + (th'q')_i - (th'q')_{i-1}); the large
            // reference values never enter a difference
            const T dth = th[0] - th[-1], dq = qv[0] - qv[-1];
            return (dth + T(0.608) * (r[6] * dq + r[7] * dth + (th[0] * qv[0] - th[-1] * qv[-1]))) / r[5];
        }
    };
    const int ka = k0 + wid * R;
    if (ka > d.nz - 2) return;
    T um = su(ka - 1, -1), u0 = su(ka - 1, 0), up = su(ka - 1, 1);   // the row below
    T w1 = sw(ka), w2 = sw(ka + 1);
    T Wm = T(0.25) * (w1 + sw(ka - 1)), W = T(0.25) * (w2 + w1);     // Wu at faces ka-1, ka
    T fz = zflux(ka - 1, T(0.25) * (sw(ka - 1) + sw(ka - 2)), Wm, W);
    T D = thv_dx(ka - 1);
#pragma unroll 1
    for (int j = 0; j < R; j++) {
        const int k = ka + j;
        if (k > d.nz - 2) break;   // uniform over the warp
        const T* r = row(k);
        const size_t id = d.at(i, k);
        T oz = T(0), ob = T(0);
        if (point && !a.ab.first) {   // the previous tendencies, in flight during the fluxes
            oz = a.hz_o[id];
            ob = a.hb_o[id];
        }
        // x face (i+1/2, k)
        const T vm = su(k, -1), v0 = su(k, 0), vp = su(k, 1);
        const T* z = zeta + at(k);
        T U = T(0.25) * (v0 + u0), z1 = z[0], z2 = z[1];
        if (wrap) {
            const int e = d.nx - 2;
            U = T(0.25) * (r[0] * (a.u[d.at(e + 1, k)] + a.u[d.at(e, k)]) + row(k - 1)[0] * (a.u[d.at(e + 1, k - 1)] + a.u[d.at(e, k - 1)]));
            z1 = a.zeta[d.at(e, k)];
            z2 = a.zeta[d.at(e + 1, k)];
        }
        const Face<T> F = face_of(xhi && k <= d.nz - 3, U, T(1), T(0.25) * (vm + um), T(1), T(0.25) * (vp + up));
        const T fu = face_flux(F, z2 - z1, z1 - z[-1], z[2] - z2, z2 + z1);
        um = vm;
        u0 = v0;
        up = vp;
        // z face (i, k+1/2)
        const T w3 = k + 2 <= d.nz - 1 ? sw(k + 2) : T(0);
        const T Wp = T(0.25) * (w3 + w2);
        const T fk = zflux(k, Wm, W, Wp);
        Wm = W;
        W = Wp;
        w2 = w3;
        const T px = (fu - __shfl_up_sync(0xffffffffu, fu, 1)) * r[2], pz = (fk - fz) * r[3];
        fz = fk;
        // Bouyancy (Buoyancy.cpp:25-48)
        const T Dk = thv_dx(k);
        const T *qc = &S.v[5][0][c] + at(k), *qr = &S.v[6][0][c] + at(k);
        const T b = r[4] * T(0.5) * (Dk + D) * T(a.c.rdx);
        const T bc = r[4] * (T(0.5) * (qc[0] + qc[-VX]) - T(0.5) * (qc[-1] + qc[-VX - 1])) * T(a.c.rdx);
        const T br = r[4] * (T(0.5) * (qr[0] + qr[-VX]) - T(0.5) * (qr[-1] + qr[-VX - 1])) * T(a.c.rdx);
        D = Dk;
        if (!point) continue;
        const T tz = -px - pz, tb = b + (-bc - br);
        if (a.ab.first) {
            a.hz_o[id] = oz = tz;
            a.hb_o[id] = ob = tb;
        }
        a.hz_n[id] = tz;
        a.hb_n[id] = tb;
        T zp = z[0] + dt15 * tz - dt05 * oz;
        zp += (dt15 * tb) - (dt05 * ob);
        store_westdown(a.zetap, d, i, k, zp);
    }
}
// Blocks a SM: what shared memory holds at launch_pzeta's rows a thread.
template <typename T, int R>
__global__ void __launch_bounds__(kTileLanes* kTileWarps, 4)
    k_pzeta(const __grid_constant__ FieldMaps<7> maps, PZetaArgs<T> a) {
    k_pzeta_body<T, R>(maps, a);
}

// ---------------------------------------------------------------------------
// Scalar advection (Advection_thermo, Advection.cpp:25-81) of th, qv, qc, qr,
// rain sedimentation (Advection_qrVT, Advection.cpp:153-192), the surface
// precipitation diagnostic (Iteration.cpp:114-119) and the per-block partial
// sums of NegativeValueProcess (MicroPhysics.cpp:116-138). Writes the raw
// interior future values; Kessler's kernel (routine calls: k_apply) finishes
// them.

enum : int { F_TH = 1, F_QV = 2, F_QC = 4, F_QR = 8 };

template <typename T>
struct PAdvArgs {
    Dims d;
    Consts c;
    Profiles p;
    const T *u, *w;
    const T* now[4];   // th, qv, qc, qr
    T* fut[4];         // thp, qvp, qcp, qrp
    T* hn[4];          // d*_advect new slot
    T* ho[4];          // d*_advect old slot
    T *hvt_n, *hvt_o;  // dqr_VT
    T* precip;         // [nx]
    double* partial;   // [gridDim.x*gridDim.y][6]: (pos, neg) of qv, qc, qr
    int* err;          // device error word (kStageErrWait), may be null
    int nvp_mask;      // F_* fields whose NVP sums are wanted
    int do_precip;     // surface rain diagnostic (with F_QR)
    AB2 ab;
};

// Final sums of NegativeValueProcess and its rescaling factor
// (MicroPhysics.cpp:125-127): nvp[2f] = 1 if positives are rescaled,
// nvp[2f+1] = 1 - |neg/pos|. One block (k_nvp_final); fixed summation
// order. `sh`: 32 * 6 doubles. (Finishing the sums in the producer's last
// block instead costs every block of the producer a fence and an atomic
// before it retires, more than this launch.)
__device__ __forceinline__ void nvp_finish(const double* partial, int nblocks, double* nvp, double* sh) {
    const int nt = blockDim.x * blockDim.y, tid = threadIdx.x + blockDim.x * threadIdx.y;
    double s[6] = {0, 0, 0, 0, 0, 0};
    // four partials a round in flight (a few round trips to L2, not one a partial)
    int b = tid;
    for (; b + 3 * nt < nblocks; b += 4 * nt) {
        double x[4][6];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int j = 0; j < 6; j++) x[q][j] = __ldcg(partial + (size_t)(b + q * nt) * 6 + j);
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int j = 0; j < 6; j++) s[j] += x[q][j];
    }
    for (; b < nblocks; b += nt)
#pragma unroll
        for (int j = 0; j < 6; j++) s[j] += __ldcg(partial + (size_t)b * 6 + j);
    block_sum(s, sh);
    if (tid == 0) {
        for (int f = 0; f < 3; f++) {
            const double pos = s[2 * f], neg = s[2 * f + 1];
            const bool skip = (pos == 0. || fabs(neg) > pos);
            nvp[2 * f] = skip ? 0.0 : 1.0;
            nvp[2 * f + 1] = skip ? 1.0 : 1. - fabs(neg / pos);
        }
    }
}

__global__ void k_nvp_final(const double* partial, int nblocks, double* nvp);

// Tile of k_padv: 31 x 8R cells a block of 32 x 8 threads, R rows a thread.
// th, qv, qc, qr, u and w are staged into shared memory with two halo cells a
// side (one TMA box a field, issued first) and the rows' coefficients beside
// them. A lane evaluates the x face west of its cell once, the velocity part
// for all fields, and takes the east flux from the next lane (the last lane
// owns no cell); going up its rows it carries each field's z flux, so a face
// between two of its rows is evaluated once too. Of the two square roots of a
// face's bracket (Advection.cpp:40-50) the wind's sign leaves one that is not
// zero, so one is taken; flux divergences multiply by r2d / rhou of the row
// instead of dividing (two roundings either way); a sedimentation flux of no
// rain needs no pow. The sums of NegativeValueProcess are reduced once for a
// thread's R cells.
// Bound by instruction issue: 35 us at 2048 x 256 FP64 and 89 at 8192 x 256,
// from 51 and 179 with two roots, a division a term, every flux through shared
// memory and a reduction a cell (FP32 44 -> 23).
template <typename T, int R>
struct PAdvShared {
    static constexpr int BZ = tile_rows(R), VZ = BZ + 4;
    T v[6][VZ][kTileVX];     // th, qv, qc, qr, u, w: each box a multiple of 128 bytes
    // rows k0-1 .. k0+BZ+1: rhou, rhow, r2dx / rhou, r2dzc / rhou, vt_c1,
    // vt_fac; mixed, of th0 and qv0: 2 ref, s0, g0, d0
    T row[BZ + 3][kPert<T> ? 14 : 6];
    double red[kTileWarps][6];
};

// MASK: the F_* fields advected; NVP sums and the precipitation go with it
// (a.nvp_mask, a.do_precip). maps: the tensor maps of th, qv, qc, qr, u, w,
// read where they lie (a kernel parameter, or global memory for a grouped
// launch): TMA takes their addresses.
template <typename T, int MASK, int R>
__device__ __forceinline__ void k_padv_body(const FieldMaps<6>& maps, const PAdvArgs<T>& a) {
    using Sh = PAdvShared<T, R>;
    constexpr int BZ = Sh::BZ, VZ = Sh::VZ, VX = kTileVX, AL = 16 / sizeof(T);
    extern __shared__ __align__(128) unsigned char padv_smem[];
    __shared__ uint64_t stage_bar;
    Sh& S = *reinterpret_cast<Sh*>(padv_smem);
    const Dims& d = a.d;
    const int lane = threadIdx.x, wid = threadIdx.y, tid = lane + kTileLanes * wid;
    const int i0 = 1 + blockIdx.x * kTileBX, k0 = 1 + blockIdx.y * BZ;
    const int x0 = (i0 - 2) & ~(AL - 1);
    const int i = i0 + lane;

    // Points outside the array read as zero; a face reads its outer neighbours
    // only where the bracket applies (2 <= index <= n-3).
    const uint32_t bar = smem_u32(&stage_bar);
    if (tid == 0) mbar_init1(bar);
    __syncthreads();
    if (tid == 0) {
        constexpr int nf = ((MASK >> 0) & 1) + ((MASK >> 1) & 1) + ((MASK >> 2) & 1) + ((MASK >> 3) & 1) + 2;
        mbar_expect_tx(bar, nf * VZ * VX * sizeof(T));
#pragma unroll
        for (int f = 0; f < 6; f++)
            if (f >= 4 || (MASK & (1 << f))) tma_load_2d(smem_u32(&S.v[f][0][0]), &maps.m[f], x0, k0 - 2, bar);
    }
    for (int t = tid; t < BZ + 3; t += kTileLanes * kTileWarps) {
        const int k = k0 - 1 + t;
        if (k > d.nz - 1) break;
        T* r = S.row[t];
        r[0] = T(a.p.rhou[k]);
        r[1] = T(a.p.rhow[k]);
        r[2] = T(a.c.r2dx) / r[0];
        r[3] = T(a.p.r2dzc[k]) / r[0];
        r[4] = T(a.p.vt_c1[k]);
        r[5] = T(a.p.vt_fac[k]);
        if constexpr (kPert<T>) {
#pragma unroll
            for (int f = 0; f < 2; f++) {
                r[6 + f] = T(2.0 * a.p.ref[f][k]);
                r[8 + f] = T(a.p.s0[f][k]);
                r[10 + f] = T(a.p.g0[f][k]);
                r[12 + f] = T(a.p.d0[f][k]);
            }
        }
    }
    const bool ok = mbar_wait_bounded(bar, 0);
    if (__syncthreads_or(!ok)) {   // the copies never landed: report and leave
        if (tid == 0 && a.err) atomicOr(a.err, kStageErrWait);
        mbar_wait_bounded(bar, 0);
        return;
    }

    const int c = i0 - x0 + lane;                 // the lane's column in the tile
    const bool cell = lane < kTileBX && i <= d.nx - 2;
    const bool wrap = (i == d.nx - 1);            // the east face of cell nx-2: the halo copy of face 1
    const bool xhi = i >= 2 && i <= d.nx - 3;
    constexpr bool vt = (MASK & F_QR) != 0;       // sedimentation goes with qr
    const T dt15 = T(1.5 * a.c.dt), dt05 = T(0.5 * a.c.dt);
    const T* const u = &S.v[4][0][0];
    const T* const w = &S.v[5][0][0];
    // z fluxes of the fields and of the rain's fall at face k (between rows
    // k-1 and k); none at the top face (Advection.cpp:57-58, :170-171)
    T fz[4] = {T(0), T(0), T(0), T(0)}, gz = T(0);
    auto zfaces = [&](int k, T (&f4)[4], T& g) {
        const int r = k - k0 + 2, at = r * VX + c;
        const T* q = S.row[k - k0 + 1];
        const bool hi = xhi && k >= 2 && k <= d.nz - 3;
        Face<T> F{};
        const bool top = k > d.nz - 2;
        if (!top) {
            const T wk = w[at];
            F = face_of(hi, q[1] * wk, S.row[k - k0][1], w[at - VX], S.row[k - k0 + 2][1], w[at + VX]);
        }
#pragma unroll
        for (int f = 0; f < 4; f++) {
            if (!(MASK & (1 << f))) continue;
            const T* v = &S.v[f][0][0] + at;
            const T vmm = v[-2 * VX], vm = v[-VX], v0 = v[0], vp = v[VX];
            T dd = v0 - vm, dm = vm - vmm, dp = vp - v0;
            if (kPert<T> && f < 2 && hi) {   // third-order differences with the profile's (mixed step)
                dd += q[12 + f];
                dm += S.row[k - k0][12 + f];
                dp += S.row[k - k0 + 2][12 + f];
            }
            f4[f] = top ? T(0) : face_flux(F, dd, dm, dp, v0 + vm);
            if (f == 3) {
                const T sm = v0 + vm;
                g = T(0);
                if (!top && sm != T(0)) {   // Advection.cpp:165-166
                    const T VT = T(1E-2) * (T(3634) * pow(q[4] * sm, T(0.1346)) * q[5]);
                    g = q[1] * VT * sm;
                }
            }
        }
    };

    double sums[6] = {0, 0, 0, 0, 0, 0};
    const int ka = k0 + wid * R;
    if (ka <= d.nz - 2) zfaces(ka, fz, gz);
#pragma unroll 1
    for (int j = 0; j < R; j++) {
        const int k = ka + j;
        if (k > d.nz - 2) break;   // uniform over the warp
        const int at = (k - k0 + 2) * VX + c;
        const size_t id = d.at(i, k);
        const T* q = S.row[k - k0 + 1];
        T o[4], ovt = T(0);
        if (cell && !a.ab.first) {   // the previous tendencies, in flight during the fluxes
#pragma unroll
            for (int f = 0; f < 4; f++)
                if (MASK & (1 << f)) o[f] = a.ho[f][id];
            if (vt) ovt = a.hvt_o[id];
        }
        // x face west of the cell (or, at nx-1, face 1, from where it lies)
        const Face<T> F = face_of(xhi && k >= 2 && k <= d.nz - 3, q[0] * (wrap ? a.u[d.at(1, k)] : u[at]), q[0], u[at - 1], q[0], u[at + 1]);
        T fu[4], zu[4], gu;
#pragma unroll
        for (int f = 0; f < 4; f++) {
            if (!(MASK & (1 << f))) continue;
            const T* v = &S.v[f][0][0] + at;
            T vm = v[-1], v0 = v[0];
            if (wrap) {
                vm = a.now[f][d.at(0, k)];
                v0 = a.now[f][d.at(1, k)];
            }
            fu[f] = face_flux(F, v0 - vm, vm - v[-2], v[1] - v0, v0 + vm);
        }
        zfaces(k + 1, zu, gu);
#pragma unroll
        for (int f = 0; f < 4; f++) {
            if (!(MASK & (1 << f))) continue;
            const T fe = __shfl_down_sync(0xffffffffu, fu[f], 1);
            T px = (fe - fu[f]) * q[2], pz = (zu[f] - fz[f]) * q[3];
            if constexpr (kPert<T>) {
                if (f < 2) {
                    // v = v0(k) + v': the v0 parts of both fluxes are added in
                    // difference form, 2 v0 (u[i+1] - u[i]) in x and
                    // s0[k+1] (m[k+1] - m[k]) + m[k] g0[k] in z, m = rhow w.
                    const T m0 = q[1] * w[at];
                    const T refz = (k == d.nz - 2) ? -m0 * q[8 + f]
                                                   : S.row[k - k0 + 2][8 + f] * (S.row[k - k0 + 2][1] * w[at + VX] - m0) + m0 * q[10 + f];
                    const T ue = (i == d.nx - 2) ? a.u[d.at(1, k)] : u[at + 1];
                    px = (fe - fu[f]) * q[2] + q[6 + f] * (ue - u[at]) * T(a.c.r2dx);
                    pz = (zu[f] - fz[f] + refz) * q[3];
                }
            }
            const T t = -px - pz;
            T tv = T(0);
            if (f == 3) tv = (gu - gz) * q[3];
            if (cell) {
                if (a.ab.first) {
                    o[f] = t;
                    a.ho[f][id] = t;
                    if (f == 3) {
                        ovt = tv;
                        a.hvt_o[id] = tv;
                    }
                }
                a.hn[f][id] = t;
                T out = S.v[f][k - k0 + 2][c] + dt15 * t - dt05 * o[f];
                if (f == 3) {
                    a.hvt_n[id] = tv;
                    out += dt15 * tv - dt05 * ovt;
                }
                a.fut[f][id] = out;
                if (f >= 1 && (a.nvp_mask & (1 << f))) {
                    double full = (double)out;
                    if (kPert<T> && f == 1) full += a.p.ref[1][k];
                    if (full >= 0.0) sums[2 * (f - 1)] += full;
                    else sums[2 * (f - 1) + 1] += full;
                }
            }
            fz[f] = zu[f];
        }
        gz = gu;
        if (a.do_precip && k == 1 && cell) {
            const T q1 = S.v[3][2][c];
            T VT = T(1E-2) * (T(3634) * pow(T(a.p.pf1) * q1, T(0.1346)) * T(a.p.pf2));
            T rain = -q[0] * (T(0.5) * (w[at + VX] + T(0)) - VT) * q1;
            a.precip[i] = (rain < T(0)) ? T(0) : rain;
        }
    }
    if (a.nvp_mask) {   // the block's sums, in a fixed order
#pragma unroll
        for (int m = 0; m < 6; m++) sums[m] = warp_sum(sums[m]);
        if (lane == 0) {
#pragma unroll
            for (int m = 0; m < 6; m++) S.red[wid][m] = sums[m];
        }
        __syncthreads();
        if (tid < 6) {
            double t = 0.0;
            for (int q = 0; q < kTileWarps; q++) t += S.red[q][tid];
            a.partial[(size_t)(blockIdx.x + gridDim.x * blockIdx.y) * 6 + tid] = t;
        }
    }
}
// Blocks a SM by shared memory at four rows a thread: three in FP64, six in FP32.
template <typename T>
constexpr int kPAdvMinBlocks = sizeof(T) == 8 ? 3 : 4;
template <typename T, int MASK, int R>
__global__ void __launch_bounds__(kTileLanes* kTileWarps, kPAdvMinBlocks<T>)
    k_padv(const __grid_constant__ FieldMaps<6> maps, PAdvArgs<T> a) {
    k_padv_body<T, MASK, R>(maps, a);
}

// ---------------------------------------------------------------------------
// Finishes th, qv, qc, qr after advection or microphysics: the rescaling of
// NegativeValueProcess, AddForcing (AddForcing.cpp:6-28) and the
// BoundaryProcess2D_center halo. One thread per interior cell.

template <typename T>
struct ApplyArgs {
    Dims d;
    Consts c;
    Profiles p;
    T* fut[4];               // thp, qvp, qcp, qrp (in place)
    const double* nvp;       // [6] from k_nvp_final
    const T* th_forcing;     // init_th_forcing (may be null)
    int mask;                // fields to finish
    int nvp_mask;            // fields to clip/rescale
    int forcing;             // add Q1LS/Q2LS
    int forcing_th;          // add dt*init_th_forcing (status_for_adding_forcing)
    int halo;                // write ghost images
};

template <typename T>
__device__ __forceinline__ T nvp_apply(T v, const double* nvp, int f) {
    if (!(v >= T(0))) return T(0);                        // MicroPhysics.cpp:121-122
    if (nvp[2 * f] != 0.0 && v > T(0)) return v * T(nvp[2 * f + 1]);   // MicroPhysics.cpp:130
    return v;
}

// What k_apply does to one value of field f at (id, row k): the rescaling of
// NegativeValueProcess, then AddForcing. Shared with the fused form at the
// top of k_kessler, so both give the same bits.
template <typename T>
struct AdvFinish {
    const double* nvp;       // [6] from k_nvp_final
    const T* th_forcing;     // init_th_forcing (may be null)
    int nvp_mask;            // fields to clip/rescale
    int forcing;             // add Q1LS/Q2LS
    int forcing_th;          // add dt*init_th_forcing
};

template <typename T>
__device__ __forceinline__ T finish_value(const AdvFinish<T>& a, const Profiles& p, T dt, int f, T v, int k,
                                          size_t id) {
    if (f >= 1 && (a.nvp_mask & (1 << f))) {
        if (kPert<T> && f == 1) {   // NegativeValueProcess acts on the full qv
            double full = p.ref[1][k] + (double)v;
            v = T(nvp_apply(full, a.nvp, 0) - p.ref[1][k]);
        } else {
            v = nvp_apply(v, a.nvp, f - 1);
        }
    }
    if (f == 0) {
        if (a.forcing) v += dt * T(p.q1ls[k]);
        if (a.forcing_th) v += dt * a.th_forcing[id];
    }
    if (f == 1 && a.forcing) v += dt * T(p.q2ls[k]);
    return v;
}

template <typename T>
__device__ __forceinline__ void k_apply_body(const ApplyArgs<T>& a) {
    const Dims& d = a.d;
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int k = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > d.nx - 2 || k > d.nz - 2) return;
    const size_t id = d.at(i, k);
    const T dt = T(a.c.dt);
    const AdvFinish<T> fin{a.nvp, a.th_forcing, a.nvp_mask, a.forcing, a.forcing_th};
    for (int f = 0; f < 4; f++) {
        if (!(a.mask & (1 << f))) continue;
        const T v = finish_value(fin, a.p, dt, f, a.fut[f][id], k, id);
        if (a.halo) store_center(a.fut[f], d, i, k, v);
        else a.fut[f][id] = v;
    }
}
template <typename T>
__global__ void k_apply(ApplyArgs<T> a) { k_apply_body<T>(a); }

// ---------------------------------------------------------------------------
// BoundaryProcess2D_all (Boundary.cpp:32-52) as a standalone pass.

template <typename T>
struct HaloArgs {
    Dims d;
    T *zetap, *w;        // westdown
    T* center[5];        // thp, u, qvp, qcp, qrp
};

template <typename T>
__global__ void k_halo_all(HaloArgs<T> a) {
    const Dims& d = a.d;
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int k = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > d.nx - 2 || k > d.nz - 2) return;
    const size_t id = d.at(i, k);
    if (k >= 2) {
        store_westdown(a.zetap, d, i, k, a.zetap[id]);
        store_westdown(a.w, d, i, k, a.w[id]);
    }
#pragma unroll
    for (int f = 0; f < 5; f++) store_center(a.center[f], d, i, k, a.center[f][id]);
}

// ---------------------------------------------------------------------------
// Kessler warm rain, applied cell by cell in the reference's order:
// autoconversion (MicroPhysics.cpp:29-51), accretion (:54-77), evaporation
// (:80-114), saturation adjustment (:7-26); then the NVP partial sums of qvp,
// qcp, qrp. One thread per interior cell.

template <typename T>
struct KesslerArgs {
    Dims d;
    Consts c;
    Profiles p;
    T *thp, *qvp, *qcp, *qrp;
    T* out[4];        // where th, qv, qc, qr go (in place, or the diffusion's inputs)
    int halo;         // write their ghost images too
    double* partial;  // NVP sums of each block
    int rows;         // rows a thread
    // The finish of the advection step (k_apply's rescaling and forcing of
    // th, qv, qc, qr) applied to each value as it is read, in place of a
    // k_apply launch.
    AdvFinish<T> pre;
    int do_pre;
};

// One cell of Kessler warm rain in compute type C.
// Cells without rain (or, for the accretion, without cloud) have rates that
// are exactly zero there, so their pow and exp are left out; lvcp = lv / (cp pib).
template <typename C>
__device__ __forceinline__ void kessler_cell(C& th, C& qv, C& qc, C& qr, C dt, C lv, C cp, C pib, C rhou,
                                             C pc, C pb, C lvcp) {
    {   // autoconversion
        C qcplus = smax(C(0), qc);
        C ar = C(0.001) * (qcplus - C(0.001));
        ar = smax(C(0), ar);
        C arcrdt = smin(ar * dt, qcplus);
        qc = qc - arcrdt;
        qr = qr + arcrdt;
    }
    {   // accretion
        C qcplus = smax(C(0), qc), qrplus = smax(C(0), qr);
        C arcrdt = C(0);
        if (qcplus != C(0) && qrplus != C(0)) {
            C cr = C(2.2) * qcplus * (pow(qrplus, C(0.875)));
            arcrdt = smin(cr * dt, qcplus);
        }
        qc = qc - arcrdt;
        qr = qr + arcrdt;
    }
    C qrplus = smax(C(0), qr);
    if (qrplus != C(0)) {   // evaporation of rain
        C qvplus = smax(C(0), qv);
        C qvs = pc * exp(C(17.27) * (pib * th - C(273.)) / (pib * th - C(36.)));
        C deficit = smax((C(1.) - qvplus / qvs), C(0.));
        C coef = C(1.6) + C(124.9) * pow((C(1E-3) * rhou * qrplus), C(0.2046));
        C er = coef * deficit * (pow(C(1E-3) * rhou * qrplus, C(0.525))) /
               ((C(5.4E5) + C(2.55E6) / (C(1E-2) * pb * qvs)) * C(1E-3) * rhou);
        C erdt = smin(qrplus, smax(C(0.), er * dt));
        qr = qr - erdt;
        qv = qv + erdt;
        th = th - lvcp * erdt;
    }
    {   // saturation adjustment
        C qvs = pc * exp(C(17.27) * (pib * th - C(273.)) / (pib * th - C(36.)));
        C tm = th * pib - C(36.);
        C phi = qvs * (C(17.27) * C(237.) * lv) / (cp * (tm * tm));
        C cnd = (qv - qvs) / (C(1) + phi);
        if (fabs(cnd) > qc && cnd < C(0)) cnd = -qc;
        qv = qv - cnd;
        qc = qc + cnd;
        th = th + lvcp * cnd;
    }
}

// The mixed step runs this kernel's arithmetic in FP64 on its FP32 storage:
// the saturation adjustment subtracts qvs from qv, which cancel to a few
// units of the FP32 epsilon near saturation.
// A block of 32 x 8 threads takes 32 columns by 8 a.rows rows, a thread a.rows
// of a column, and reduces the sums once for them. Bound by instruction issue
// and its latencies (FP64 exp, divisions; pow in rain), so registers are held
// to four blocks a SM (a few spills; 24.6, 21.9, 18.9 us at two, three, four):
// 26 -> 19 us at 2048 x 256, 81 -> 50 at 8192 x 256, with rain in a small part
// of the grid.
constexpr int kKesslerWarps = 8;
template <typename T>
__device__ __forceinline__ void k_kessler_body(const KesslerArgs<T>& a) {
    using C = double;
    __shared__ double red[kKesslerWarps][6];
    const Dims& d = a.d;
    const int lane = threadIdx.x, wid = threadIdx.y;
    const int i = 1 + blockIdx.x * 32 + lane;
    const int ka = 1 + (blockIdx.y * kKesslerWarps + wid) * a.rows;
    double sums[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int j = 0; j < a.rows; j++) {
        const int k = ka + j;
        if (k > d.nz - 2) break;   // uniform over the warp
        if (i > d.nx - 2) continue;
        const size_t id = d.at(i, k);
        const C th0 = kPert<T> ? a.p.ref[0][k] : 0.0, qv0 = kPert<T> ? a.p.ref[1][k] : 0.0;
        T tv = a.thp[id], qvv = a.qvp[id], qcv = a.qcp[id], qrv = a.qrp[id];
        if (a.do_pre) {
            const T dt = T(a.c.dt);
            tv = finish_value(a.pre, a.p, dt, 0, tv, k, id);
            qvv = finish_value(a.pre, a.p, dt, 1, qvv, k, id);
            qcv = finish_value(a.pre, a.p, dt, 2, qcv, k, id);
            qrv = finish_value(a.pre, a.p, dt, 3, qrv, k, id);
        }
        C th = th0 + (C)tv, qv = qv0 + (C)qvv, qc = qcv, qr = qrv;
        kessler_cell<C>(th, qv, qc, qr, a.c.dt, a.c.lv, a.c.cp, a.p.pib[k], a.p.rhou[k], a.p.pc[k], a.p.pb[k],
                        a.p.lvcp[k]);
        const T res[4] = {T(th - th0), T(qv - qv0), T(qc), T(qr)};
#pragma unroll
        for (int f = 0; f < 4; f++) {
            if (a.halo) store_center(a.out[f], d, i, k, res[f]);
            else a.out[f][id] = res[f];
        }
        const C q[3] = {qv, qc, qr};
#pragma unroll
        for (int f = 0; f < 3; f++) {
            if (q[f] >= C(0)) sums[2 * f] += q[f];
            else sums[2 * f + 1] += q[f];
        }
    }
    // the block's sums, in a fixed order
#pragma unroll
    for (int m = 0; m < 6; m++) sums[m] = warp_sum(sums[m]);
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < 6; m++) red[wid][m] = sums[m];
    }
    __syncthreads();
    const int tid = lane + 32 * wid;
    if (tid < 6) {
        double t = 0.0;
        for (int q = 0; q < kKesslerWarps; q++) t += red[q][tid];
        a.partial[(size_t)(blockIdx.x + gridDim.x * blockIdx.y) * 6 + tid] = t;
    }
}
template <typename T>
__global__ void __launch_bounds__(32 * kKesslerWarps, 4) k_kessler(KesslerArgs<T> a) { k_kessler_body<T>(a); }

// ---------------------------------------------------------------------------
// Eddy coefficients (Turbulence::RKM_RKH, Turbulent.cpp:5-45) with their
// center halo. One thread per interior cell.

template <typename T>
struct RKArgs {
    Dims d;
    Consts c;
    Profiles p;
    const T *u, *w, *thp;
    T *RKM, *RKH;
    unsigned* kmax;   // [2], 0 before: the largest RKM, RKH (float bits, rounded up)
};

// Raises *m to the largest of the block's values v (positive floats compared
// as their bits; a NaN's bits are above all of them). Blocks that would not
// raise it issue no atomic.
__device__ __forceinline__ void block_max_bits(unsigned v, unsigned* sh, unsigned* m) {
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    v = __reduce_max_sync(0xffffffffu, v);
    if ((tid & 31) == 0) sh[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < (int)(blockDim.x * blockDim.y) >> 5; w++) v = max(v, sh[w]);
        if (v > *(volatile unsigned*)m) atomicMax(m, v);
    }
}
__device__ __forceinline__ unsigned bits_up(double x) { return __float_as_uint(__double2float_ru(x)); }
__device__ __forceinline__ unsigned bits_up(float x) { return __float_as_uint(x); }

// R rows a thread: the rows between are loaded once, not three times, and all
// of them at once, with a barrier and an atomic for R times as many cells.
// Where the numerator of Ri is at least a quarter of a positive denominator, in
// most cells, there is no mixing and neither a division nor a root is taken; Ri
// itself decides everywhere else (whatever theta's sign, and where it is zero).
template <typename T, int R>
__device__ __forceinline__ void k_rkm_rkh_body(const RKArgs<T>& a) {
    const Dims& d = a.d;
    const int i = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int k0 = 1 + (blockIdx.y * blockDim.y + threadIdx.y) * R;
    __shared__ unsigned sh[2][32];
    unsigned kmx = 0u, khx = 0u;   // bits, above all others' where a value is NaN
    if (i <= d.nx - 2 && k0 <= d.nz - 2) {
        T u[R + 2][2], w[R + 1][3], th[R + 2];   // rows k0-1 .. k0+R; w from k0
#pragma unroll
        for (int q = 0; q < R + 2; q++) {
            const size_t e = d.at(i, min(k0 - 1 + q, d.nz - 1));
            u[q][0] = a.u[e];
            u[q][1] = a.u[e + 1];
            th[q] = a.thp[e];
            if (q)
#pragma unroll
                for (int x = 0; x < 3; x++) w[q - 1][x] = a.w[e + x - 1];
        }
#pragma unroll
        for (int q = 0; q < R; q++) {
            const int k = k0 + q;
            if (k > d.nz - 2) break;
            T Rzeta = T(0.5) * ((w[q + 1][2] + w[q][2]) - (w[q + 1][0] + w[q][0])) * T(a.c.r2dx) +
                      T(0.5) * ((u[q + 2][1] + u[q + 2][0]) - (u[q][1] + u[q][0])) * T(a.p.r2dzcc[k]);
            T rot = (u[q + 1][1] - u[q + 1][0]) * T(a.c.rdx) + (w[q + 1][1] - w[q][1]) * T(a.p.rdzc[k]);
            T th0 = th[q + 1];
            T dth = th[q + 2] - th[q];
            if constexpr (kPert<T>) {       // perturbation storage: add the profile parts
                th0 += T(a.p.ref[0][k]);
                dth += T(a.p.g0[0][k]);
            }
            const T def2 = Rzeta * Rzeta + T(2.) * (rot * rot);
            const T r2 = T(a.p.r2dzcc[k]), num = T(a.c.gravity) * dth * r2, den = th0 * def2;   // Ri = num / den
            T km = T(0.), kh = T(0.);
            if (!(den > T(0) && num >= T(0.25) * den)) {
                const T Ri = (T(a.c.gravity) / th0 * dth * r2) / def2;
                const T lam = T(a.p.lambda2[k]), ld = lam * sqrt(def2);
                if (Ri < T(0)) {
                    km = ld * sqrt(T(1.) - T(16.) * Ri);
                    kh = ld * T(1.4) * sqrt(T(1.) - T(40.) * Ri);
                } else if (T(0) < Ri && Ri < T(0.25)) {
                    const T f = T(1.) - T(4.) * Ri, f4 = (f * f) * (f * f);
                    km = ld * f4;
                    kh = ld * T(1.4) * (T(1.) - T(1.2) * Ri) * f4;
                }
            }
            const T kmax = T(a.p.kmax[k]);
            km = smin(smax(km, T(10.)), kmax);
            kh = smin(smax(kh, T(10.)), kmax);
            store_center(a.RKM, d, i, k, km);
            store_center(a.RKH, d, i, k, kh);
            kmx = max(kmx, bits_up(km));
            khx = max(khx, bits_up(kh));
        }
    }
    block_max_bits(kmx, sh[0], a.kmax);
    block_max_bits(khx, sh[1], a.kmax + 1);
}
template <typename T, int R>
__global__ void __launch_bounds__(256) k_rkm_rkh(RKArgs<T> a) { k_rkm_rkh_body<T, R>(a); }

// ---------------------------------------------------------------------------
// In-place Gauss-Seidel diffusion (Turbulence::Mparam / Hparam,
// Turbulent.cpp:68-114), exact to round-off, with the top-layer nudging of
// theta and zeta fused in (NumericalProcess.cpp:60-85).
//
// The reference sweeps k outer, i inner and reads the already-updated left
// (i-1) and lower (k-1) neighbours, so cell (i, k) obeys
//   v'(i,k) = A0(i,k) + C(i,k) v'(i,k-1) + B(i,k) v'(i-1,k),
// where A0, C and B depend on old values only: B is the left-face
// coefficient, C the lower-face one, A0 collects the rest.
//
// The recurrence is lower triangular in (k, i): a cell depends on the cells
// left of it in its row and below it in its column. The padded rows are cut
// into tiles of tr rows (from k = 1) by 128 columns (from i = 0), one warp a
// tile, 4 cells a lane. A pass computes every tile at once from inflows left
// by the previous pass: the value left of each of its rows (the right outflow
// of the tile on its left) and the row below it (the top outflow of the tile
// below). Inside a tile each row is exact: a scan over the warp of the affine
// maps y_i = a_i + B_i y_{i-1}, a_i = A0 + C x (x the value below), the
// lanes' maps composed with shuffles, then applied cell by cell from the
// inflow.
//
// A tile's outputs are final once its inflows are, so the tiles of the d-th
// anti-diagonal (b + c = d) are final after pass d + 1, and nb + nc - 1 passes
// reproduce the sequential sweep over the tiles. The passes stop earlier, as
// soon as no outflow that another tile reads changed bit for bit from one
// pass to the next: the following pass would then read the same inflows and
// repeat every value, so that is the fixed point the full count reaches. A
// pass shrinks an inflow's error by about B + C. These passes are the schedule
// for large coefficients alone: with those a step normally has (1e-3) the
// single pass below (k_gs_sweep) gives the sweep to round-off, and none of
// these runs unless it asks for them.
//
// Pass 1 reads the old values: it forms A0 from them and stores it, takes
// its inflows from them (the guess), and writes no field, so every tile of it
// reads the old state. Passes 2 on read A0, form B and C from the eddy
// coefficients (which no pass changes) and write the field; at least two
// passes run.
//
// Buffers (parity q = pass & 1 written by a pass, q ^ 1 read):
//   right[q][f][b][c][r]   y at the tile's last column, rows r = 0..tr-1
//   top[q][f][b][c][col]   y of the tile's top row, col = 0..127
// The last block of a pass (a thread-fence and counter, no waiting) decides
// whether another pass follows, and sets the condition of the graph's WHILE
// node when the passes run in a graph; the last pass of a sweep resets the
// pass state for the next one (the host's loop also clears it first). In a
// graph they are the body of a conditional node that k_gs_sweep opens: the
// inputs and pass 1 the first time round, a later pass each time; a pass that
// finds the sweep converged returns at once.

template <typename T>
struct GSArgs {
    Dims d;
    Consts c;
    Profiles p;
    T* v[5];          // zetap (Mparam, RKM), thp, qvp, qcp, qrp (Hparam, RKH)
    const T *RKM, *RKH;
    int mask;         // bit f: diffuse field f
    int nudge;        // fuse Nudge_theta (field 1) and Nudge_zeta (field 0)
    T* A0;            // per-cell constant term, [5][cells] (written by pass 1 / k_gs_coeffs)
    T *C, *B;         // per-cell lower and left coefficients (the cluster schedule only)
    int* err;         // device error word (kGSErrWait, the cluster schedule), may be null
};

constexpr int kGSMaxNX = 8192;
constexpr int kGSMaxPerThread = 8;      // cells a thread of the cal_u column integral

constexpr int kGTCols = 128;   // columns of a tile: 32 lanes x 4 cells
constexpr int kGTPer = 4;
// Rows of a tile: the autotuner's knob (the passes a sweep needs do not
// depend on it; taller tiles mean fewer, longer tiles a pass).
constexpr int kGSTileRowsMin = 4, kGSTileRowsMax = 32, kGSTileRowsDefault = 8;
constexpr int kGSRowVals = 9;   // scalars a tile row keeps in shared memory
inline bool gs_tile_rows_ok(int tr) { return tr == 4 || tr == 8 || tr == 16 || tr == 32; }
// Blocks a SM the tile kernel is compiled for: three in FP64 (up to 168
// registers a thread: pass 1 then keeps its rolling windows without spilling;
// the 1360 tiles of the 2048 x 256 default still fit in one wave), four in
// FP32.
template <typename T>
constexpr int kGSTileMinBlocks = sizeof(T) == 8 ? 3 : 4;

struct GSTileCtl {    // zero before a sweep
    int pass;         // passes of the sweep completed
    int changed[2];   // by parity of the pass that wrote an outflow differing from its previous one
    int done;         // blocks of the current pass that finished
    int more;         // another pass follows (read by the host loop)
    int passes;       // passes run by the last sweep
};

template <typename T>
struct GSTileArgs {
    int nb, nc, tr;   // bands of tr rows from k = 1, chunks of 128 columns from i = 0
    T* right;         // [2][5][nb][nc][tr]
    T* top;           // [2][5][nb][nc][128]
    GSTileCtl* ctl;
    long long* exec;  // kernels run inside graph loops (counted by the deciding block)
    __device__ __forceinline__ size_t ri(int q, int f, int b, int c) const {
        return ((((size_t)q * 5 + f) * nb + b) * nc + c) * tr;
    }
    __device__ __forceinline__ size_t ti(int q, int f, int b, int c) const {
        return ((((size_t)q * 5 + f) * nb + b) * nc + c) * kGTCols;
    }
};

// 4 consecutive cells of one row (16-byte aligned: i a multiple of 4, rows of
// a multiple of 32 cells).
template <typename T>
__device__ __forceinline__ void gs_ld4(const T* p, T (&x)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 u = __ldg(reinterpret_cast<const float4*>(p));
        x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w;
    } else {
        const double2 u = __ldg(reinterpret_cast<const double2*>(p)), w = __ldg(reinterpret_cast<const double2*>(p) + 1);
        x[0] = u.x, x[1] = u.y, x[2] = w.x, x[3] = w.y;
    }
}

// One pass over every tile: 4 warps (tiles) a block. Each lane keeps its
// cells' rows of K (k-1, k and, in pass 1, k+1) and, in pass 1, of the old
// field (k, k+1) in registers, rolled up a row at a time; the next row's
// loads are issued before the current row's scan. Left and right neighbours
// come from the adjacent lane by shuffle (the tile's edge lanes load theirs).
// B, C (and in pass 1 A0) follow Turbulent.cpp:83-88 for zeta and :107-112
// for the scalars term by term. The ghost i = 0 gets the constant map
// v'(0, k) = v(0, k) (never updated), cells beyond NX the identity map, so a
// row's scan needs no edge cases. Stores the nudged values (Nudge_zeta,
// Nudge_theta) of interior cells, carries the un-nudged ones.
// FIRST: pass 1 (launched on its own, before the loop of the later passes).
template <typename T, bool FIRST>
__device__ __forceinline__ void k_gs_tiles_body(const GSArgs<T>& a, const GSTileArgs<T>& t, cudaGraphConditionalHandle h) {
    __shared__ int any_changed;
    // per warp and row of its tile: cz, the czd and czu density factors,
    // nudging dn and tn, the inflow left of the row and its previous value,
    // and (pass 1, th' and qv') the profile differences at k and k+1
    __shared__ T rowv[4][kGSTileRowsMax][kGSRowVals];
    const Dims& d = a.d;
    const int NX = d.nx - 2, kend = d.nz - 2;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) any_changed = 0;
    __syncthreads();
    constexpr bool first = FIRST;
    // a pass launched after the sweep converged has nothing to do, nor has
    // pass 1 once the passes have begun (a loop body launches both kernels)
    if (FIRST ? t.ctl->pass != 0 : !*(volatile int*)&t.ctl->more) return;
    const int pass = FIRST ? 1 : t.ctl->pass + 1;
    const int q = pass & 1, qp = q ^ 1;
    const int tile = blockIdx.x * 4 + wid;
    const int ntiles = 5 * t.nb * t.nc;
    const int c = tile % t.nc, b = (tile / t.nc) % t.nb, f = tile / (t.nc * t.nb);
    if (tile < ntiles && (a.mask & (1 << f))) {   // uniform over the warp
        T* v = a.v[f];
        const bool mom = (f == 0);
        const T* K = mom ? a.RKM : a.RKH;
        T* A0s = a.A0 + (size_t)f * d.cells();
        const int i0 = c * kGTCols + lane * kGTPer;
        const bool act = i0 < d.pitch;   // pitch is a multiple of 32, so of kGTPer
        const int k0 = 1 + b * t.tr;
        const int rows = min(t.tr, kend - k0 + 1);
        const int ilast = c * kGTCols + kGTCols - 1;   // the tile's last column
        const bool edge_l = (lane == 0 && i0 >= 1);             // its left neighbour is in another tile
        const bool edge_r = (lane == 31 && act && i0 + 3 <= NX); // its right neighbour is needed
        const T cx = T(a.c.rdx2 * a.c.dt);
        const bool pert = kPert<T> && (f == 1 || f == 2);
        auto row4 = [&](const T* base, int k, T (&x)[4]) {
            if (act) gs_ld4(base + d.at(i0, k), x);
            else x[0] = x[1] = x[2] = x[3] = T(0);
        };
        bool diff = false;
        // the row below the tile: the old row 0 (never updated), or the top
        // outflow of the tile below (pass 1: the old values there)
        T below[kGTPer];
        if (b == 0 || first) {
            row4(v, k0 - 1, below);
            if (b == 0) {
#pragma unroll
                for (int e = 0; e < kGTPer; e++)
                    if (!(i0 + e >= 1 && i0 + e <= NX)) below[e] = T(0);
            }
        } else {
#pragma unroll
            for (int e = 0; e < kGTPer; e++) below[e] = t.top[t.ti(qp, f, b - 1, c) + lane * kGTPer + e];
        }
        // rolling windows: K rows k-1 (Kd), k (Kc), k+1 (Ku); old field rows k (v0), k+1 (vu)
        T Kd[4], Kc[4], Ku[4], v0[4], vu[4], An[4];
        row4(K, k0 - 1, Kd);
        row4(K, k0, Kc);
        if (first) {
            row4(K, k0 + 1, Ku);
            row4(v, k0, v0);
            row4(v, k0 + 1, vu);
        } else {
            row4(A0s, k0, An);
        }
        // the edge lanes' neighbours in the next tiles, a row ahead as well:
        // lane 0 K(i0-1, k) (and, rolled, K(i0-1, k-1)); lane 31 in pass 1
        // K(i0+4, k) and v(i0+4, k)
        T eKl = T(0), eKld = T(0), eKr = T(0), evr = T(0);
        if (edge_l) {
            eKl = K[d.at(i0 - 1, k0)];
            eKld = K[d.at(i0 - 1, k0 - 1)];
        }
        if (first && edge_r) {
            eKr = K[d.at(i0 + 4, k0)];
            evr = v[d.at(i0 + 4, k0)];
        }
        const T* rin = t.right + t.ri(qp, f, b, c - 1);   // read only when c > 0
        T* rout = t.right + t.ri(q, f, b, c);
        const T* rold = t.right + t.ri(qp, f, b, c);
        // the rows' scalars, one lane a row, all loads at once
        if (lane < rows) {
            const int k = k0 + lane;
            T* rv = rowv[wid][lane];
            if (mom) {
                rv[0] = T(a.p.gsM_cz[k]);
                rv[1] = T(a.p.gsM_rhod[k]);
                rv[2] = T(a.p.rhou[k]);
            } else {
                rv[0] = T(a.p.gsS_cz[k]);
                rv[1] = T(a.p.gsS_rhod[k]);
                rv[2] = T(a.p.rhow[k + 1]);
            }
            T dn = T(0), tn = T(0);   // nudging of row k: out = y - dn (y - tn)
            if (a.nudge && f == 0) dn = T(a.p.dtcgr_zeta[k]);
            if (a.nudge && f == 1) {
                dn = T(a.p.dtcgr_th[k]);
                tn = kPert<T> ? T(-a.p.dn[0][k]) : T(a.p.thb_init[k]);
            }
            rv[3] = dn;
            rv[4] = tn;
            rv[5] = (c > 0) ? (first ? v[d.at(c * kGTCols - 1, k)] : rin[lane]) : T(0);
            rv[6] = (c + 1 < t.nc) ? (first ? v[d.at(ilast, k)] : rold[lane]) : T(0);
            if (first && pert) {
                rv[7] = T(a.p.d0[f - 1][k]);
                rv[8] = T(a.p.d0[f - 1][k + 1]);
            }
        }
        __syncwarp();
        for (int r = 0; r < rows; r++) {
            const T* rv = rowv[wid][r];
            const int k = k0 + r;
            const bool more_rows = r + 1 < rows;
            // the next row's loads, in flight during this row's work
            T Kn[4], vn[4], An2[4];
            T eKl_n = T(0), eKr_n = T(0), evr_n = T(0);
            if (more_rows) {
                if (first) {
                    row4(K, k + 2, Kn);
                    row4(v, k + 2, vn);
                } else {
                    row4(K, k + 1, Kn);
                    row4(A0s, k + 1, An2);
                }
                if (edge_l) eKl_n = K[d.at(i0 - 1, k + 1)];
                if (first && edge_r) {
                    eKr_n = K[d.at(i0 + 4, k + 1)];
                    evr_n = v[d.at(i0 + 4, k + 1)];
                }
            }
            // neighbours across lanes (the edge lanes' from the next tiles)
            T Kl0 = __shfl_up_sync(0xffffffffu, Kc[3], 1);
            T Kld0 = __shfl_up_sync(0xffffffffu, Kd[3], 1);
            T Kr3 = __shfl_down_sync(0xffffffffu, Kc[0], 1);
            T vr3 = __shfl_down_sync(0xffffffffu, first ? v0[0] : T(0), 1);
            if (edge_l) {
                Kl0 = eKl;
                Kld0 = eKld;
            }
            if (first && edge_r) {
                Kr3 = eKr;
                vr3 = evr;
            }
            const T cz = rv[0], rhod = rv[1], rhou_ = rv[2];
            T aa[kGTPer], bb[kGTPer];
#pragma unroll
            for (int e = 0; e < kGTPer; e++) {
                const int i = i0 + e;
                T A0, B, C;
                if (!act || i > NX) {          // beyond NX: identity
                    A0 = T(0);
                    B = T(1);
                    C = T(0);
                } else if (i == 0) {           // the ghost: constant map
                    A0 = first ? v0[0] : An[0];
                    B = T(0);
                    C = T(0);
                } else {
                    const T Kl = (e == 0) ? Kl0 : Kc[e - 1];
                    T ax = T(0), bx, czu = T(0), czd;
                    if (mom) {
                        const T Kld = (e == 0) ? Kld0 : Kd[e - 1];
                        bx = T(0.5) * (Kl + Kld);
                        czd = rhod * T(0.5) * (Kd[e] + Kld);
                        if (first) {
                            ax = T(0.5) * (Kc[e] + Kd[e]);
                            czu = rhou_ * T(0.5) * (Kc[e] + Kl);
                        }
                    } else {
                        bx = T(0.5) * (Kc[e] + Kl);
                        czd = rhod * T(0.5) * (Kc[e] + Kd[e]);
                        if (first) {
                            const T Kr = (e == 3) ? Kr3 : Kc[e + 1];
                            ax = T(0.5) * (Kr + Kc[e]);
                            czu = rhou_ * T(0.5) * (Ku[e] + Kc[e]);
                        }
                    }
                    C = cz * czd;
                    B = cx * bx;
                    if (first) {
                        const T vc = v0[e], vr = (e == 3) ? vr3 : v0[e + 1];
                        T du = vu[e] - vc, dd = vc;
                        if (pert) {   // th', qv' about a profile
                            du += rv[8];
                            dd += rv[7];
                        }
                        // v + cx (ax (vr - v) - bx (v - v'[i-1])) + cz (czu du - czd (dd - v'below))
                        A0 = vc + cx * (ax * (vr - vc) - bx * vc) + cz * (czu * du - czd * dd);
                    } else {
                        A0 = An[e];
                    }
                }
                if (first && act) A0s[d.at(i0, k) + e] = A0;
                aa[e] = A0 + C * below[e];
                bb[e] = B;
            }
            // the lane's map over its cells: y_out = P + M y_in
            T P = T(0), M = T(1);
#pragma unroll
            for (int e = 0; e < kGTPer; e++) {
                P = aa[e] + bb[e] * P;
                M = bb[e] * M;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {   // inclusive scan: own map after the lower lanes'
                const T qP = __shfl_up_sync(0xffffffffu, P, o), qM = __shfl_up_sync(0xffffffffu, M, o);
                if (lane >= o) {
                    P = P + M * qP;
                    M = M * qM;
                }
            }
            // the inflow left of the row (chunk 0 starts at the ghost, B = 0)
            const T x = rv[5];
            const T eP = __shfl_up_sync(0xffffffffu, P, 1), eM = __shfl_up_sync(0xffffffffu, M, 1);
            T y = (lane == 0) ? x : eP + eM * x;
            const T dn = rv[3], tn = rv[4];
            T out[kGTPer];
#pragma unroll
            for (int e = 0; e < kGTPer; e++) {
                y = aa[e] + bb[e] * y;
                below[e] = y;
                out[e] = y - dn * (y - tn);
            }
            if (act && !first) {
                T* dst = v + d.at(i0, k);
                if (i0 >= 1 && i0 + kGTPer - 1 <= NX) {
                    if constexpr (sizeof(T) == 4) {
                        *reinterpret_cast<float4*>(dst) = make_float4(out[0], out[1], out[2], out[3]);
                    } else {
                        *reinterpret_cast<double2*>(dst) = make_double2(out[0], out[1]);
                        *reinterpret_cast<double2*>(dst + 2) = make_double2(out[2], out[3]);
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < kGTPer; e++)
                        if (i0 + e >= 1 && i0 + e <= NX) dst[e] = out[e];
                }
            }
            const T yr = __shfl_sync(0xffffffffu, y, 31);   // y at the tile's last column
            if (lane == 0) {
                rout[r] = yr;
                if (c + 1 < t.nc && !(yr == rv[6])) diff = true;   // read by the tile on the right
            }
            // roll the windows up a row
            if (more_rows) {
                eKld = eKl;
                eKl = eKl_n;
                eKr = eKr_n;
                evr = evr_n;
#pragma unroll
                for (int e = 0; e < kGTPer; e++) {
                    Kd[e] = Kc[e];
                    if (first) {
                        Kc[e] = Ku[e];
                        Ku[e] = Kn[e];
                        v0[e] = vu[e];
                        vu[e] = vn[e];
                    } else {
                        Kc[e] = Kn[e];
                        An[e] = An2[e];
                    }
                }
            }
        }
        T* tout = t.top + t.ti(q, f, b, c) + lane * kGTPer;
        const T* told = t.top + t.ti(qp, f, b, c) + lane * kGTPer;
        const int ktop = k0 + rows - 1;
#pragma unroll
        for (int e = 0; e < kGTPer; e++) {
            tout[e] = below[e];
            if (b + 1 < t.nb) {   // read by the tile above
                const T prev = first ? (act ? v[d.at(i0 + e, ktop)] : T(0)) : told[e];
                if (!(below[e] == prev)) diff = true;
            }
        }
        if (__any_sync(0xffffffffu, diff) && lane == 0) any_changed = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (any_changed) t.ctl->changed[q] = 1;
        __threadfence();
        const int prev = atomicAdd(&t.ctl->done, 1);
        if (prev == (int)gridDim.x - 1) {   // the last block of the pass decides
            __threadfence();
            const int ch = *(volatile int*)&t.ctl->changed[q];
            // pass 1 writes no field: a second pass always follows; every tile
            // is final after nb + nc - 1 passes
            const int more = (first || ch) && pass < max(2, t.nb + t.nc - 1);
            t.ctl->done = 0;
            t.ctl->passes = pass;
            t.ctl->more = more;
            if (more) {
                t.ctl->changed[qp] = 0;   // the next pass writes that parity
                t.ctl->pass = pass;
            } else {                      // ready for the next sweep
                t.ctl->changed[0] = t.ctl->changed[1] = 0;
                t.ctl->pass = 0;
            }
            if (t.exec) *t.exec += 1;
            if (h) cudaGraphSetConditional(h, more ? 1u : 0u);
        }
    }
}
template <typename T, bool FIRST>
__global__ void __launch_bounds__(128, kGSTileMinBlocks<T>) k_gs_tiles(GSArgs<T> a, GSTileArgs<T> t, cudaGraphConditionalHandle h) { k_gs_tiles_body<T, FIRST>(a, t, h); }

// ---------------------------------------------------------------------------
// The same recurrence in one pass, for the coefficients a step normally has.
//
// With beta the largest B + C of the grid, an error of a cell's inflow is
// beta^n of itself n cells later, so a tile needs no exact inflow: started
// hz rows below and 16 cells left of the cells it owns, from the old values
// (which differ from the new ones by beta times the field's local change), its
// owned cells are off by beta^(hz+1) of that change. hz is the least number of
// rows that puts this below 2^-56 (FP32: 2^-28), from the largest eddy
// coefficient of the grid (k_rkm_rkh), usually 4 to 8; where more than
// kGWHaloMax would be needed (B + C above about 0.1, FP32 0.3) the kernel
// writes nothing and asks for the repeated passes above instead; so does a
// tile that has met an infinity or NaN, which no tail outruns (whatever its
// rows hold of these is still there in the last one). Along a row
// the same bound cuts the scan short: y left of a lane's four cells is the
// lanes' offsets of the 8 (B <= 2^-7, FP32 2^-3.5) or 16 cells before it.
//
// The fields are read from one set of arrays and written to another, so every
// tile sees the old values whatever the others have done; qv, qc and qr may
// still lack the rescaling of NegativeValueProcess, which is then applied as
// they are read (no pass of its own). Ghost cells are copied.
//
// One warp a tile of tr rows by 108 owned columns (27 lanes of 4 cells; four
// halo lanes on the left, one on the right for the explicit terms), for zeta
// and pairs of scalars (which share the coefficients: least work), or for one
// field (shorter rows: least time where the grid has few tiles). Rows arrive
// by cp.async kGWDepth ahead, each lane reading back only what it copied, so
// no barrier is needed. Bound by the instruction issue of the few warps a
// scheduler holds (2048 x 256 FP64: 6.1 M warp instructions over 912 tiles of 22
// rows, 306 a row, ~4 cycles each at one warp a scheduler). Measured at 2048 x 256 against the
// three passes it replaces: 32 / 91 us FP64, 19 / 63 us FP32; 8192 x 256 FP64
// 81 / 260, 128 x 64 12.6 / 81. A form that makes the rows' coefficients by
// other warps first (shared memory, a barrier every 8 or 16 rows) took 34 us
// and 90 us at the two large FP64 grids and 13.7 us at the small one.
constexpr int kGWOwnLanes = 27, kGWLeft = 4, kGWOwn = 4 * kGWOwnLanes;
constexpr int kGWRowsMax = 32, kGWHaloMax = 16, kGWDepth = 4, kGWWarps = 2;
template <typename T>
constexpr float kGWBits = sizeof(T) == 8 ? 56.f : 28.f;

template <typename T>
struct GSSweepArgs {
    Dims d;
    Consts c;
    Profiles p;
    const T* src[5];     // zeta, th, qv, qc, qr before the diffusion, ghosts included
    T* dst[5];
    const T *RKM, *RKH;
    const double* nvp;   // rescaling of qv, qc, qr still to do (k_nvp_final's), or null
    int nudge;           // fuse Nudge_theta (field 1) and Nudge_zeta (field 0)
    int nb, nc, tr;      // bands of tr rows from k = 1, chunks of kGWOwn columns from i = 0
    int jobs;            // 3: zeta; th, qv; qc, qr. 5: every field on its own
    const unsigned* kmax;
    float fz[2];         // largest C / K over the rows: Mparam, Hparam
    GSTileCtl* ctl;      // more: the repeated passes are needed (0 before)
    // a captured step that puts its rare loops at its end (run_step_direct):
    // the solve's check has failed; set when the end has to run (0 before)
    const int* solve_more;
    int* redo;
};

// Asks for the repeated passes (ctl->more), and for the end of a captured step.
template <typename T>
__device__ __forceinline__ void gs_ask(const GSSweepArgs<T>& a, bool passes, cudaGraphConditionalHandle h) {
    if (passes) a.ctl->more = 1;
    if (a.redo) *a.redo = 1;
    if (h) cudaGraphSetConditional(h, 1u);
}

template <typename T>
struct GSSweepShared {
    T ring[kGWDepth][4][128];            // K, then the job's fields (a power of two a slot)
    T row[kGWRowsMax + kGWHaloMax][8];   // per row: lower and upper factors, nudging (dn, tn), profile differences
};

// The rescaling of field f (2, 3, 4): nvp_apply's with its factor taken as 1
// where it does not rescale.
__device__ __forceinline__ double gs_factor(const double* nvp, int f) {
    return nvp[2 * (f - 2)] != 0.0 ? nvp[2 * (f - 2) + 1] : 1.0;
}
template <typename T>
__device__ __forceinline__ T gs_finish(T fac, T v) { return v >= T(0) ? v * fac : T(0); }

// The tile's constants and rolling windows; one lane's part of a row is its
// four cells.
template <typename T, bool MOM, int NF>
struct GSSweepTile {
    static constexpr int D = kGWDepth;
    int i0, NX, f0, lane;
    bool act, edge, own, wide;
    size_t pitch;
    const T* from[1 + NF];   // the next row to copy: K, then the fields
    T* to[NF];               // the next row to store
    T fac[NF];               // rescaling of each field (gs_factor)
    bool fin[NF];            // it is still to do
    T cx;
    T Kp[4], Kc[4], lo[4], v0[NF][4], below[NF][4], klp;

    __device__ __forceinline__ T* slot(GSSweepShared<T>& S, int q, int arr) const {
        return &S.ring[q][arr][sizeof(T) == 8 ? 2 * lane : 4 * lane];
    }
    // copies the next row of K and the fields into slot q
    __device__ __forceinline__ void issue(GSSweepShared<T>& S, int q, bool on) {
        if (act && on) {
#pragma unroll
            for (int arr = 0; arr <= NF; arr++) {
                T* dst = slot(S, q, arr);
                cp_async16(dst, from[arr]);
                if constexpr (sizeof(T) == 8) cp_async16(dst + 64, from[arr] + 2);
                from[arr] += pitch;
            }
        }
        cp_async_commit();
    }
    __device__ __forceinline__ static void read4(const T* s, T (&x)[4]) {
        if constexpr (sizeof(T) == 8) {
            const double2 u = *reinterpret_cast<const double2*>(s), w = *reinterpret_cast<const double2*>(s + 64);
            x[0] = u.x, x[1] = u.y, x[2] = w.x, x[3] = w.y;
        } else {
            const float4 u = *reinterpret_cast<const float4*>(s);
            x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w;
        }
    }
    // the row in slot q (level k), finished; then the slot's next row
    __device__ __forceinline__ void take(GSSweepShared<T>& S, const GSSweepArgs<T>& a, int q, int k, bool more, T (&Kx)[4],
                                         T (&vx)[NF][4]) {
        cp_async_wait<D - 1>();
        read4(slot(S, q, 0), Kx);
#pragma unroll
        for (int f = 0; f < NF; f++) {
            read4(slot(S, q, 1 + f), vx[f]);
            if (!MOM && fin[f]) {
                const bool full = kPert<T> && f0 + f == 2;
                const double ref = full ? a.p.ref[1][k] : 0.0, fd = full ? gs_factor(a.nvp, 2) : 0.0;
#pragma unroll
                for (int e = 0; e < 4; e++)
                    vx[f][e] = full ? T(gs_finish(fd, ref + (double)vx[f][e]) - ref) : gs_finish(fac[f], vx[f][e]);
            }
        }
        issue(S, q, more);
    }
    __device__ __forceinline__ void store4(int f, const T (&x)[4]) const {
        if constexpr (sizeof(T) == 8) {
            *reinterpret_cast<double2*>(to[f]) = make_double2(x[0], x[1]);
            *reinterpret_cast<double2*>(to[f] + 2) = make_double2(x[2], x[3]);
        } else {
            *reinterpret_cast<float4*>(to[f]) = make_float4(x[0], x[1], x[2], x[3]);
        }
    }

    // Row k: its K above (Ku) and fields above (vu) arrive, its results go to
    // `below` and, when asked for, to memory; the windows move up a row.
    __device__ __forceinline__ void row(const T* rv, const T (&Ku)[4], const T (&vu)[NF][4], bool store) {
        const T fd = rv[0], fu = rv[1];
        // left, right, lower and upper coefficients (Turbulent.cpp:83-88, :107-112)
        T B[4], R[4], C[4], U[4];
        const T kl = __shfl_up_sync(0xffffffffu, Kc[3], 1);
        if constexpr (MOM) {
            T g = kl + klp;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const T up = Kc[e] + (e ? Kc[e - 1] : kl);
                B[e] = cx * g;
                g = Kc[e] + Kp[e];
                R[e] = cx * g;
                C[e] = fd * lo[e];
                U[e] = fu * up;
                lo[e] = up;
            }
            klp = kl;
        } else {
            const T kr = __shfl_down_sync(0xffffffffu, Kc[0], 1);
            T g = Kc[0] + kl;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const T up = Ku[e] + Kc[e];
                B[e] = cx * g;
                g = (e < 3 ? Kc[e + 1] : kr) + Kc[e];
                R[e] = cx * g;
                C[e] = fd * lo[e];
                U[e] = fu * up;
                lo[e] = up;
            }
        }
        if (edge) {   // ghosts and padding keep their values
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (i0 + e < 1 || i0 + e > NX) B[e] = R[e] = C[e] = U[e] = T(0);
        }
        const T M = (B[0] * B[1]) * (B[2] * B[3]);
        T M2 = T(0);
        if (wide) M2 = M * __shfl_up_sync(0xffffffffu, M, 1);
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const T vr = __shfl_down_sync(0xffffffffu, v0[f][0], 1);
            // y itself, A0 + C y_below + B y_left, added up in the passes'
            // order; in FP32 zeta's increment y - v, whose terms are all
            // small beside v: one rounding at v's size a step, not four.
            constexpr bool kInc = kPert<T> && MOM;
            T vl = T(0);
            if constexpr (kInc) vl = __shfl_up_sync(0xffffffffu, v0[f][3], 1);
            T x[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const T v = v0[f][e], right = e < 3 ? v0[f][e + 1] : vr;
                T du = vu[f][e] - v, dd = v;
                if (kPert<T> && !MOM && f0 + f <= 2) {   // th', qv' about a profile
                    du += rv[5 + 2 * f];
                    dd += rv[4 + 2 * f];
                }
                if constexpr (kInc)
                    x[e] = (R[e] * (right - v) + B[e] * ((e ? v0[f][e - 1] : vl) - v)) + (U[e] * du + C[e] * (below[f][e] - dd));
                else
                    x[e] = v + (R[e] * (right - v) - B[e] * v) + (U[e] * du - C[e] * dd) + C[e] * below[f][e];
            }
            // the lane's offset with no inflow, then the lanes' before it
            T P = ((x[0] * B[1] + x[1]) * B[2] + x[2]) * B[3] + x[3];
            T q = __shfl_up_sync(0xffffffffu, P, 1);
            if (lane >= 1) P += M * q;
            if (wide) {
                q = __shfl_up_sync(0xffffffffu, P, 2);
                if (lane >= 2) P += M2 * q;
            }
            T y = __shfl_up_sync(0xffffffffu, P, 1);
            if (lane == 0) y = kInc ? T(0) : v0[f][0];
            T out[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                y = x[e] + B[e] * y;
                out[e] = kInc ? v0[f][e] + y : y;
                below[f][e] = out[e];
            }
            if ((MOM || (f == 0 && f0 == 1)) && rv[2] != T(0)) {   // Nudge_zeta, Nudge_theta
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (i0 + e >= 1 && i0 + e <= NX) out[e] = out[e] - rv[2] * (out[e] - rv[3]);
            }
            if (store) {
                if (own) store4(f, out);
                to[f] += pitch;
            }
#pragma unroll
            for (int e = 0; e < 4; e++) v0[f][e] = vu[f][e];
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            Kp[e] = Kc[e];
            Kc[e] = Ku[e];
        }
    }
};

// False where the tile has met a value that is not finite.
template <typename T, bool MOM, int NF>
__device__ __forceinline__ bool gs_sweep_tile(const GSSweepArgs<T>& a, GSSweepShared<T>& S, int f0, int b, int c, int hz,
                                              bool wide) {
    constexpr int D = kGWDepth;
    const Dims& d = a.d;
    const GSBand band = gs_band(b, a.tr, hz, d.nz);
    const int k0 = band.k0, kl = band.kl, ks = band.ks;
    GSSweepTile<T, MOM, NF> t;
    t.lane = threadIdx.x & 31;
    t.f0 = f0;
    t.NX = d.nx - 2;
    t.pitch = d.pitch;
    t.i0 = c * kGWOwn + 4 * (t.lane - kGWLeft);
    t.act = t.i0 >= 0 && t.i0 < d.pitch;
    t.edge = t.i0 < 1 || t.i0 + 3 > t.NX;
    t.own = t.act && t.lane >= kGWLeft && t.lane < kGWLeft + kGWOwnLanes;
    t.wide = wide;
    t.cx = T(0.5) * T(a.c.rdx2 * a.c.dt);
    t.from[0] = (MOM ? a.RKM : a.RKH) + d.at(t.i0, ks - 1);
#pragma unroll
    for (int f = 0; f < NF; f++) {
        t.from[1 + f] = a.src[f0 + f] + d.at(t.i0, ks - 1);
        t.to[f] = a.dst[f0 + f] + d.at(t.i0, k0);
        t.fin[f] = !MOM && a.nvp && f0 + f >= 2;
        t.fac[f] = t.fin[f] ? T(gs_factor(a.nvp, f0 + f)) : T(1);
    }
    if (!t.act) {   // lanes outside the array: zeros
        for (int q = 0; q < D; q++)
            for (int arr = 0; arr <= NF; arr++)
                for (int e = 0; e < (sizeof(T) == 8 ? 2 : 4); e++) {
                    t.slot(S, q, arr)[e] = T(0);
                    if (sizeof(T) == 8) t.slot(S, q, arr)[64 + e] = T(0);
                }
    }
    const int n = kl - ks + 3;   // rows to copy: ks-1 .. kl+1
#pragma unroll
    for (int q = 0; q < D; q++) t.issue(S, q, q < n);
    for (int r = t.lane; r <= kl - ks; r += 32) {   // the rows' scalars
        const int k = ks + r;
        T* rv = S.row[r];
        const T cz = MOM ? T(a.p.gsM_cz[k]) : T(a.p.gsS_cz[k]);
        rv[0] = cz * (T(0.5) * (MOM ? T(a.p.gsM_rhod[k]) : T(a.p.gsS_rhod[k])));
        rv[1] = cz * (T(0.5) * (MOM ? T(a.p.rhou[k]) : T(a.p.rhow[k + 1])));
        T dn = T(0), tn = T(0);   // out = y - dn (y - tn)
        if (a.nudge && f0 == 0) dn = T(a.p.dtcgr_zeta[k]);
        if (a.nudge && f0 == 1) {
            dn = T(a.p.dtcgr_th[k]);
            tn = kPert<T> ? T(-a.p.dn[0][k]) : T(a.p.thb_init[k]);
        }
        rv[2] = dn;
        rv[3] = tn;
        if (kPert<T> && !MOM) {   // th', qv': their profiles' differences
#pragma unroll
            for (int f = 0; f < NF; f++)
                if (f0 + f <= 2) {
                    rv[4 + 2 * f] = T(a.p.d0[f0 + f - 1][k]);
                    rv[5 + 2 * f] = T(a.p.d0[f0 + f - 1][k + 1]);
                }
        }
    }
    __syncwarp();
    t.take(S, a, 0, ks - 1, D < n, t.Kp, t.below);
    if (band.bottom && t.own) {   // the ghost row under the grid
#pragma unroll
        for (int f = 0; f < NF; f++) {
            t.to[f] -= t.pitch;
            t.store4(f, t.below[f]);
            t.to[f] += t.pitch;
        }
    }
    t.take(S, a, 1, ks, D + 1 < n, t.Kc, t.v0);
    t.klp = T(0);
    if constexpr (MOM) {
        t.klp = __shfl_up_sync(0xffffffffu, t.Kp[3], 1);
        t.lo[0] = t.Kp[0] + t.klp;
#pragma unroll
        for (int e = 1; e < 4; e++) t.lo[e] = t.Kp[e] + t.Kp[e - 1];
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) t.lo[e] = t.Kc[e] + t.Kp[e];
    }
    // not unrolled: a tile runs few rows, and fetching four times the code
    // costs more than the moves it would save (13 rows: 14.8 against 12.6 us)
    int q = 2;
#pragma unroll 1
    for (int k = ks; k <= kl; k++) {
        T Ku[4], vu[NF][4];
        t.take(S, a, q, k + 1, k + D < kl + 1, Ku, vu);
        q = (q + 1) & (D - 1);
        t.row(S.row[k - ks], Ku, vu, k >= k0);
    }
    if (band.top && t.own) {   // the ghost row over the grid
#pragma unroll
        for (int f = 0; f < NF; f++) t.store4(f, t.v0[f]);
    }
    cp_async_wait<0>();
    bool finite = true;
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int e = 0; e < 4; e++) finite = finite && isfinite(t.below[f][e]);
    return __all_sync(0xffffffffu, finite);
}

template <typename T>
__device__ __forceinline__ void k_gs_sweep_body(const GSSweepArgs<T>& a, cudaGraphConditionalHandle h) {
    __shared__ __align__(16) GSSweepShared<T> S[kGWWarps];
    const float cx = (float)(a.c.rdx2 * a.c.dt);
    const float km = __uint_as_float(a.kmax[0]), kh = __uint_as_float(a.kmax[1]);
    // bits an inflow error loses a cell, with a little to spare for the roundings here
    const float l = -log2f(1.001f * fmaxf(km * (cx + a.fz[0]), kh * (cx + a.fz[1])));
    const float lx = -log2f(1.001f * cx * fmaxf(km, kh));
    const int hz = max(1, (int)ceilf(kGWBits<T> / l) - 1);
    const bool ok = km == km && kh == kh && l > 0.f && hz <= kGWHaloMax && 16.f * lx >= kGWBits<T>;
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0)
        if (!ok || (a.solve_more && *a.solve_more)) gs_ask(a, !ok, h);
    if (!ok) return;
    const int wid = threadIdx.x >> 5;
    const int tile = blockIdx.x * kGWWarps + wid;
    if (tile >= a.jobs * a.nb * a.nc) return;
    const int c = tile % a.nc, b = (tile / a.nc) % a.nb, job = tile / (a.nc * a.nb);
    const bool wide = 8.f * lx < kGWBits<T>;
    bool finite;
    if (job == 0) finite = gs_sweep_tile<T, true, 1>(a, S[wid], 0, b, c, hz, wide);
    else if (a.jobs == 3) finite = gs_sweep_tile<T, false, 2>(a, S[wid], 2 * job - 1, b, c, hz, wide);
    else finite = gs_sweep_tile<T, false, 1>(a, S[wid], job, b, c, hz, wide);
    if (!finite && (threadIdx.x & 31) == 0) gs_ask(a, true, h);
}
template <typename T>
__global__ void __launch_bounds__(32 * kGWWarps) k_gs_sweep(GSSweepArgs<T> a, cudaGraphConditionalHandle h) { k_gs_sweep_body<T>(a, h); }

// The inputs of the repeated passes, which run in place: src, finished, copied
// to dst (ghosts too). Nothing to do once a sweep's passes have begun.
template <typename T>
__device__ __forceinline__ void k_gs_inputs_body(const GSSweepArgs<T>& a) {
    if (a.ctl->pass != 0) return;
    const Dims& d = a.d;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= d.nx || k >= d.nz) return;
    const size_t id = d.at(i, k);
    T v[5];   // all loads before the first store, which might change them for all the compiler knows
#pragma unroll
    for (int f = 0; f < 5; f++) v[f] = a.src[f][id];
#pragma unroll
    for (int f = 0; f < 5; f++) {
        if (a.nvp && f >= 2) {
            if (kPert<T> && f == 2) v[f] = T(gs_finish(gs_factor(a.nvp, 2), a.p.ref[1][k] + (double)v[f]) - a.p.ref[1][k]);
            else v[f] = gs_finish(T(gs_factor(a.nvp, f)), v[f]);
        }
    }
#pragma unroll
    for (int f = 0; f < 5; f++) a.dst[f][id] = v[f];
}
template <typename T>
__global__ void k_gs_inputs(GSSweepArgs<T> a) { k_gs_inputs_body<T>(a); }

// ---------------------------------------------------------------------------
// The second schedule of the same recurrence: one thread-block cluster a field.
// k_gs_coeffs forms A0, C, B for every cell of the five fields in parallel;
// k_gs_cluster then runs the recurrence, one cluster per field. Row k is a
// first-order linear recurrence along i (v'(0,k) the untouched ghost), solved
// as a scan of affine maps: each thread composes the maps of its PER
// contiguous cells and the warp scans those with shuffles; warps pass the
// carry along the row to the next warp, so consecutive warps work on
// consecutive rows at the same time (a wavefront across the cluster). One
// pass and no repeated arithmetic: the schedule for many cases stepping at
// once (a batch), where the GPU is busy with other cases while a cluster's
// chain runs; the tiles are for one case alone, where the chain is the
// step's critical path. Results agree with the tiles' to round-off (the
// carries associate differently).

// A0, C, B of cell (i, k) of field blockIdx.z, i = 0..pitch-1, k = 1..nz-2
// (Turbulent.cpp:83-88 for zeta, :107-112 for the scalars). The ghost i = 0
// gets the constant map v'(0, k) = v(0, k) (never updated), cells beyond
// NX the identity map, so a row's scan needs no edge cases.
template <typename T>
__global__ void k_gs_coeffs(GSArgs<T> a) {
    const int f = blockIdx.z;
    if (!(a.mask & (1 << f))) return;
    const Dims& d = a.d;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= d.pitch || k > d.nz - 2) return;
    const T* v = a.v[f];
    if (i == 0 || i > d.nx - 2) {
        const size_t e = (size_t)f * d.cells() + d.at(i, k);
        a.A0[e] = (i == 0) ? v[d.at(0, k)] : T(0);
        a.C[e] = T(0);
        a.B[e] = (i == 0) ? T(0) : T(1);
        return;
    }
    const bool mom = (f == 0);
    const T* K = mom ? a.RKM : a.RKH;
    const T cx = T(a.c.rdx2 * a.c.dt);
    const T cz = mom ? T(a.p.gsM_cz[k]) : T(a.p.gsS_cz[k]);
    T v0 = v[d.at(i, k)], vr = v[d.at(i + 1, k)], vu = v[d.at(i, k + 1)];
    T ax, bx, czu, czd;
    if (mom) {
        T Kc = K[d.at(i, k)], Kd = K[d.at(i, k - 1)], Kl = K[d.at(i - 1, k)], Kld = K[d.at(i - 1, k - 1)];
        ax = T(0.5) * (Kc + Kd);
        bx = T(0.5) * (Kl + Kld);
        czu = T(a.p.rhou[k]) * T(0.5) * (Kc + Kl);
        czd = T(a.p.gsM_rhod[k]) * T(0.5) * (Kd + Kld);
    } else {
        T Kc = K[d.at(i, k)], Kr = K[d.at(i + 1, k)], Kl = K[d.at(i - 1, k)];
        T Ku = K[d.at(i, k + 1)], Kd = K[d.at(i, k - 1)];
        ax = T(0.5) * (Kr + Kc);
        bx = T(0.5) * (Kc + Kl);
        czu = T(a.p.rhow[k + 1]) * T(0.5) * (Ku + Kc);
        czd = T(a.p.gsS_rhod[k]) * T(0.5) * (Kc + Kd);
    }
    T du = vu - v0, dd = v0;
    if (kPert<T> && (f == 1 || f == 2)) {   // th', qv' about a profile
        du += T(a.p.d0[f - 1][k + 1]);
        dd += T(a.p.d0[f - 1][k]);
    }
    // v + cx (ax (vr - v) - bx (v - v'[i-1])) + cz (czu du - czd (dd - v'below))
    const size_t e = (size_t)f * d.cells() + d.at(i, k);
    a.A0[e] = v0 + cx * (ax * (vr - v0) - bx * v0) + cz * (czu * du - czd * dd);
    a.C[e] = cz * czd;
    a.B[e] = cx * bx;
}

constexpr int kGSSpinLimit = 1 << 22;   // polls before a wait gives up
constexpr int kGSErrWait = 1;           // device error word: a Gauss-Seidel wait gave up
constexpr size_t kGSRingBytes = 200 * 1024;   // cp.async ring of coefficient rows
constexpr int kGSCarry = 64;            // inbox slots (rows) of a warp
constexpr int kGSAckEvery = 16;         // rows between acknowledgements

// Flags between CTAs of a cluster: acquire / release at cluster scope through
// generic addresses (local shared memory, or a peer CTA's mapped into the
// cluster window).
__device__ __forceinline__ int ld_acquire_cluster(const int* p) {
    int v;
    asm volatile("ld.acquire.cluster.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cluster(int* p, int v) {
    asm volatile("st.release.cluster.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_cluster_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.cluster.b64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_cluster_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.cluster.b64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// A carry travels as row-tagged 64-bit words: (row << 32) | 32 bits of the
// value (one word for float, two for double). A 64-bit store is seen whole,
// so a reader that finds its row in every word holds that row's value; no
// flag and no fence is needed.
template <typename T>
struct Tagged {
    static constexpr int kWords = sizeof(T) / 4;
    __device__ static void put(unsigned long long* w, T x, int row) {
        const unsigned long long tag = (unsigned long long)(unsigned)row << 32;
        if constexpr (sizeof(T) == 4) {
            st_relaxed_cluster_u64(w, tag | __float_as_uint(x));
        } else {
            const unsigned long long b = (unsigned long long)__double_as_longlong(x);
            st_relaxed_cluster_u64(w, tag | (b >> 32));
            st_relaxed_cluster_u64(w + 1, tag | (b & 0xffffffffull));
        }
    }
    // true and x set when every word carries `row`
    __device__ static bool get(const unsigned long long* w, int row, T& x) {
        const unsigned long long w0 = ld_relaxed_cluster_u64(w);
        if ((int)(w0 >> 32) != row) return false;
        if constexpr (sizeof(T) == 4) {
            x = __uint_as_float((unsigned)w0);
        } else {
            const unsigned long long w1 = ld_relaxed_cluster_u64(w + 1);
            if ((int)(w1 >> 32) != row) return false;
            x = __longlong_as_double((long long)((w0 << 32) | (w1 & 0xffffffffull)));
        }
        return true;
    }
};

// The recurrence of one field spread over a cluster of CS CTAs. The padded
// row is cut into chunks of 32*PER cells, one per warp; global warp g sits in
// CTA g / W as its warp g % W (W warps a CTA). Each warp walks the rows in
// order on its own: it waits for the carry-in that warp g-1 left, row-tagged,
// in its own inbox (written locally, or into this CTA's shared memory from
// the previous CTA through the cluster window), acknowledges every
// kGSAckEvery-th row in warp g-1's shared memory (a release store, so its
// reads of the inbox come first), and, once warp g+1 has acknowledged the row
// that last used the inbox slot it is about to reuse, writes its carry-out
// into warp g+1's inbox. Everything is polled in local shared memory. Cluster barriers open (all inboxes
// initialised before any peer writes) and close (no CTA exits while a peer may
// still write into it) the kernel. Each wait polls at most kGSSpinLimit
// times; a warp that gives up raises the abort flag of every CTA of the
// cluster and the device error word, so every wait ends. Coefficient rows are
// staged in shared memory by cp.async, D rows ahead (a thread reads back only
// what it copied); the rows' nudging scalars are tabulated in shared memory at
// the start. Dynamic shared memory: D * 3 * blockDim.x * PER values of T, then
// 2 * nz values of T.
constexpr int kGSClusterWarps = 10;   // warps a CTA at most (NX = 8192: 9)

// The carry of a row pair: two row-tagged values (the pair's first row as tag).
template <typename T>
struct Tagged2 {
    static constexpr int kWords = 2 * Tagged<T>::kWords;
    __device__ static void put(unsigned long long* w, T x0, T x1, int row) {
        Tagged<T>::put(w, x0, row);
        Tagged<T>::put(w + Tagged<T>::kWords, x1, row);
    }
    __device__ static bool get(const unsigned long long* w, int row, T& x0, T& x1) {
        return Tagged<T>::get(w, row, x0) && Tagged<T>::get(w + Tagged<T>::kWords, row, x1);
    }
};

// Two rows a step. With V_i = (v'(i, k), v'(i, k+1)) the pair obeys
// V_i = alpha_i + M_i V_{i-1}, M_i = [[B_k, 0], [C_{k+1} B_k, B_{k+1}]],
// alpha_i = (a_i, A0_{k+1} + C_{k+1} a_i), a_i = A0_k + C_k v'(i, k-1): one scan
// over the row advances both rows, so the serial chain has half as many
// steps, each with five values a shuffle round instead of two (the rounds'
// shuffles are independent and overlap). The cells are then applied with the
// scalar formulas, row k first. An odd last row runs as a pair whose second
// row is the identity and is not stored.
template <typename T, int PER, int D, int CS>
__global__ void __cluster_dims__(CS, 1, 1) __launch_bounds__(32 * kGSClusterWarps) k_gs_cluster(GSArgs<T> a) {
    static_assert(D % 2 == 0, "the ring holds whole row pairs");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kW = Tagged2<T>::kWords;
    __shared__ unsigned long long inbox[kGSClusterWarps][kGSCarry][kW];
    __shared__ int ack_in[kGSClusterWarps], abort_flag;
    namespace cgx = cooperative_groups;
    cgx::cluster_group cl = cgx::this_cluster();
    const int crank = (int)cl.block_rank();
    const int f = blockIdx.x / CS;
    const Dims& d = a.d;
    const int NX = d.nx - 2, kend = d.nz - 2;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, W = blockDim.x >> 5;
    for (int j = tid; j < kGSClusterWarps * kGSCarry * kW; j += blockDim.x)
        (&inbox[0][0][0])[j] = 0ull;    // tag 0: no row
    if (tid < kGSClusterWarps) ack_in[tid] = 0;
    if (tid == 0) abort_flag = 0;
    // nudging of row k: out = x - dn[k] (x - tn[k]) (dn = 0: none)
    T* dn_tab = reinterpret_cast<T*>(smem_raw) + (size_t)D * 3 * blockDim.x * PER;
    T* tn_tab = dn_tab + d.nz;
    for (int k = tid; k < d.nz; k += blockDim.x) {
        T dn = T(0), tn = T(0);
        if (a.nudge && f == 0) dn = T(a.p.dtcgr_zeta[k]);                      // Nudge_zeta
        if (a.nudge && f == 1) {                                                 // Nudge_theta
            dn = T(a.p.dtcgr_th[k]);
            tn = kPert<T> ? T(-a.p.dn[0][k]) : T(a.p.thb_init[k]);
        }
        dn_tab[k] = dn;
        tn_tab[k] = tn;
    }
    cl.sync();
    const int gwn = (d.pitch + 32 * PER - 1) / (32 * PER);   // warps with cells
    const int g = crank * W + wid;
    const bool run = (a.mask & (1 << f)) && g < gwn;
    if (run) {
        T* v = a.v[f];
        const int i0 = (g * 32 + lane) * PER;
        const bool act = i0 < d.pitch;       // pitch is a multiple of PER
        const size_t fo = (size_t)f * d.cells();
        const T* gsrc[3] = {a.A0 + fo, a.C + fo, a.B + fo};
        T* ring = reinterpret_cast<T*>(smem_raw);
        constexpr int kVec = 16 / sizeof(T);
        auto slot = [&](int r, int arr) { return ring + ((size_t)(r * 3 + arr) * blockDim.x + tid) * PER; };
        auto issue = [&](int k, int r) {
            if (act && k <= kend) {
#pragma unroll
                for (int arr = 0; arr < 3; arr++) {
                    const T* src = gsrc[arr] + d.at(i0, k);
                    T* dst = slot(r, arr);
#pragma unroll
                    for (int q = 0; q < PER; q += kVec) cp_async16(dst + q, src + q);
                }
            }
            cp_async_commit();
        };
        // neighbours in the chain and their flags
        const bool has_pred = g > 0, has_succ = g + 1 < gwn;
        const int pc = (g - 1) / W, pw = (g - 1) % W, sc = (g + 1) / W, sw = (g + 1) % W;
        int* pred_ack = has_pred ? cl.map_shared_rank(&ack_in[pw], pc) : nullptr;
        unsigned long long* succ_box = has_succ ? cl.map_shared_rank(&inbox[sw][0][0], sc) : nullptr;
        auto give_up = [&]() {   // lane 0 of a warp whose wait ran out: stop the cluster
            for (int r = 0; r < CS; r++) *(volatile int*)cl.map_shared_rank(&abort_flag, r) = 1;
            if (a.err) atomicOr(a.err, kGSErrWait);
        };
        auto wait_carry = [&](int k, T& x0, T& x1) {   // all lanes; warp-uniform result
            bool okw = false;
            const unsigned long long* w = &inbox[wid][k % kGSCarry][0];
            for (int it = 0; it < kGSSpinLimit; it++) {
                if (Tagged2<T>::get(w, k, x0, x1)) {
                    okw = true;
                    break;
                }
                if (*(volatile int*)&abort_flag) break;
            }
            const bool all = __all_sync(0xffffffffu, okw);
            if (!all && lane == 0 && !*(volatile int*)&abort_flag) give_up();
            return all;
        };
        auto wait_ge = [&](const int* p, int target) {   // all lanes; warp-uniform result
            bool okw = false;
            for (int it = 0; it < kGSSpinLimit; it++) {
                if (ld_acquire_cluster(p) >= target) {
                    okw = true;
                    break;
                }
                if (*(volatile int*)&abort_flag) break;
            }
            const bool all = __all_sync(0xffffffffu, okw);
            if (!all && lane == 0 && !*(volatile int*)&abort_flag) give_up();
            return all;
        };
        T vdn[PER];
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int i = i0 + e;
            vdn[e] = (act && i >= 1 && i <= NX) ? v[d.at(i, 0)] : T(0);
        }
#pragma unroll
        for (int r = 0; r < D; r++) issue(1 + r, r);
        bool ok = true;
        int ack_seen = 0;   // last acknowledgement read from warp g+1
        auto pair = [&](int k, int r) {   // rows k and k+1 (k+1 may be past the last row)
            const bool two = k + 1 <= kend;
            const T dn0 = dn_tab[k], tn0 = tn_tab[k];
            const T dn1 = two ? dn_tab[k + 1] : T(0), tn1 = two ? tn_tab[k + 1] : T(0);
            const int s = k % kGSCarry;
            // read the carry-in early: when warp g-1 is ahead it is there
            T x0 = T(0), x1 = T(0);   // warp 0 starts at the ghost's constant map
            bool have = !has_pred || Tagged2<T>::get(&inbox[wid][s][0], k, x0, x1);
            cp_async_wait<D - 2>();
            T Aa[PER], Bk[PER], A2[PER], C2[PER], B2[PER];
            if (act) {
                const T* sa = slot(r, 0);
                const T* scc = slot(r, 1);
                const T* sb = slot(r, 2);
                const T* ta = slot(r + 1, 0);
                const T* tc = slot(r + 1, 1);
                const T* tb = slot(r + 1, 2);
#pragma unroll
                for (int e = 0; e < PER; e++) {
                    Aa[e] = sa[e] + scc[e] * vdn[e];
                    Bk[e] = sb[e];
                    A2[e] = two ? ta[e] : T(0);
                    C2[e] = two ? tc[e] : T(0);
                    B2[e] = two ? tb[e] : T(1);
                }
            } else {
#pragma unroll
                for (int e = 0; e < PER; e++) {
                    Aa[e] = T(0);
                    Bk[e] = T(1);
                    A2[e] = T(0);
                    C2[e] = T(0);
                    B2[e] = T(1);
                }
            }
            // the lane's map over its cells: (p0, p1) offsets, M = [[m00, 0], [m10, m11]]
            T p0 = T(0), p1 = T(0), m00 = T(1), m10 = T(0), m11 = T(1);
#pragma unroll
            for (int e = 0; e < PER; e++) {
                const T c0 = Aa[e], c1 = A2[e] + C2[e] * Aa[e];
                const T n00 = Bk[e], n10 = C2[e] * Bk[e], n11 = B2[e];
                p1 = c1 + n10 * p0 + n11 * p1;
                p0 = c0 + n00 * p0;
                m10 = n10 * m00 + n11 * m10;
                m00 = n00 * m00;
                m11 = n11 * m11;
            }
            issue(k + D, r);
            issue(k + 1 + D, r + 1);
            T s0 = p0, s1 = p1, s00 = m00, s10 = m10, s11 = m11;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const T q0 = __shfl_up_sync(0xffffffffu, s0, o), q1 = __shfl_up_sync(0xffffffffu, s1, o);
                const T q00 = __shfl_up_sync(0xffffffffu, s00, o), q10 = __shfl_up_sync(0xffffffffu, s10, o);
                const T q11 = __shfl_up_sync(0xffffffffu, s11, o);
                if (lane >= o) {   // own map after the lower lanes'
                    s1 = s1 + s10 * q0 + s11 * q1;
                    s0 = s0 + s00 * q0;
                    s10 = s10 * q00 + s11 * q10;
                    s00 = s00 * q00;
                    s11 = s11 * q11;
                }
            }
            const T t0 = __shfl_sync(0xffffffffu, s0, 31), t1 = __shfl_sync(0xffffffffu, s1, 31);
            const T t00 = __shfl_sync(0xffffffffu, s00, 31), t10 = __shfl_sync(0xffffffffu, s10, 31);
            const T t11 = __shfl_sync(0xffffffffu, s11, 31);
            T e0 = __shfl_up_sync(0xffffffffu, s0, 1), e1 = __shfl_up_sync(0xffffffffu, s1, 1);
            T e00 = __shfl_up_sync(0xffffffffu, s00, 1), e10 = __shfl_up_sync(0xffffffffu, s10, 1);
            T e11 = __shfl_up_sync(0xffffffffu, s11, 1);
            if (lane == 0) {
                e0 = T(0);
                e1 = T(0);
                e00 = T(1);
                e10 = T(0);
                e11 = T(1);
            }
            if (has_pred) {
                if (!__all_sync(0xffffffffu, have)) ok = ok && wait_carry(k, x0, x1);
                if (((k - 1) >> 1) % (kGSAckEvery / 2) == 0) {   // every kGSAckEvery rows
                    __syncwarp();
                    if (lane == 0) st_release_cluster(pred_ack, k);
                }
            }
            if (has_succ) {
                // slot s last held the pair at row k - kGSCarry
                if (ack_seen < k - kGSCarry) {
                    ok = ok && wait_ge(&ack_in[wid], k - kGSCarry);
                    ack_seen = ld_acquire_cluster(&ack_in[wid]);
                }
                if (lane == 0) Tagged2<T>::put(succ_box + (size_t)s * kW, t0 + t00 * x0, t1 + t10 * x0 + t11 * x1, k);
            }
            T y0 = e0 + e00 * x0, y1 = e1 + e10 * x0 + e11 * x1;
            T out0[PER], out1[PER];
#pragma unroll
            for (int e = 0; e < PER; e++) {
                y0 = Aa[e] + Bk[e] * y0;
                y1 = (A2[e] + C2[e] * y0) + B2[e] * y1;
                vdn[e] = y1;
                out0[e] = y0 - dn0 * (y0 - tn0);
                out1[e] = y1 - dn1 * (y1 - tn1);
            }
            auto store = [&](int kk, const T (&out)[PER]) {
                T* dst = v + d.at(i0, kk);
                if (act && i0 >= 1 && i0 + PER - 1 <= NX) {
#pragma unroll
                    for (int q = 0; q < PER; q += kVec) {
                        if constexpr (sizeof(T) == 4)
                            *reinterpret_cast<float4*>(dst + q) = make_float4(out[q], out[q + 1], out[q + 2], out[q + 3]);
                        else
                            *reinterpret_cast<double2*>(dst + q) = make_double2(out[q], out[q + 1]);
                    }
                } else if (act) {
#pragma unroll
                    for (int e = 0; e < PER; e++)
                        if (i0 + e >= 1 && i0 + e <= NX) dst[e] = out[e];
                }
            };
            store(k, out0);
            if (two) store(k + 1, out1);
        };
        for (int k = 1; k <= kend && ok; k += D) {
#pragma unroll
            for (int r = 0; r < D; r += 2)
                if (k + r <= kend && ok) pair(k + r, r);
        }
        cp_async_wait<0>();
    }
    cl.sync();
}

// ---------------------------------------------------------------------------
// Top-layer nudging as standalone passes (NumericalProcess.cpp:60-96).

template <typename T>
struct NudgeArgs {
    Dims d;
    Consts c;
    Profiles p;
    T *thp, *zetap, *qvp;
    const T* qv;
    int do_th, do_zeta;
    double tau;       // moisture_nudge_time, 0 = off
    const int* skip;  // nothing to do where *skip (may be null)
};

template <typename T>
__device__ __forceinline__ void k_nudge_body(const NudgeArgs<T>& a) {
    if (a.skip && *a.skip) return;
    const Dims& d = a.d;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= d.nx || k >= d.nz) return;
    const size_t id = d.at(i, k);
    const bool inner = (i >= 1 && i <= d.nx - 2 && k >= 1 && k <= d.nz - 2);
    if (inner && a.do_th) {
        T x = a.thp[id];
        T tref = kPert<T> ? T(-a.p.dn[0][k]) : T(a.p.thb_init[k]);
        a.thp[id] = x - T(a.p.dtcgr_th[k]) * (x - tref);
    }
    if (inner && a.do_zeta) {
        T x = a.zetap[id];
        a.zetap[id] = x - T(a.p.dtcgr_zeta[k]) * x;
    }
    if (a.tau != 0.0)  // every cell, ghosts included (NumericalProcess.cpp:90-94)
        a.qvp[id] = a.qvp[id] + T(a.c.dt) * ((kPert<T> ? T(-a.p.dn[1][k]) : T(a.p.qvb0[k])) - a.qv[id]) / T(a.tau);
}
template <typename T>
__global__ void k_nudge(NudgeArgs<T> a) { k_nudge_body<T>(a); }

// ---------------------------------------------------------------------------
// Horizontal means (Iteration::updateMean, Iteration.cpp:42-86): thb, qvb and
// thvb = thb (1 + 0.608 qvb) per level with their 1D halos. One block per
// interior level. Optionally rotates ubarTop (nextTimeStep, :166-167).

template <typename T>
struct MeanArgs {
    Dims d;
    const double *ref_th, *ref_qv;   // perturbation profiles (null in the FP64 step)
    const T *thp, *qvp;
    double *thb, *qvb, *thvb;
    double* ubar;   // [0] ubarTop, [1] ubarTopp
    int rotate_ubar;
    const int* skip;  // nothing to do where *skip (may be null)
};

template <typename T>
__device__ __forceinline__ void k_update_mean_body(const MeanArgs<T>& a) {
    __shared__ double sh[32 * 2];
    if (a.skip && *a.skip) return;
    const Dims& d = a.d;
    const int k = 1 + blockIdx.x;
    double s[2] = {0, 0};
    // eight loads in flight a thread: the rows come from L2 or memory, and a
    // loop of single loads waited for each
    const T *th = a.thp + d.at(0, k), *qv = a.qvp + d.at(0, k);
    const int step = blockDim.x;
    int i = 1 + threadIdx.x;
    for (; i + 3 * step <= d.nx - 2; i += 4 * step) {
        T x[4], y[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            x[e] = th[i + e * step];
            y[e] = qv[i + e * step];
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            s[0] += (double)x[e];
            s[1] += (double)y[e];
        }
    }
    for (; i <= d.nx - 2; i += step) {
        s[0] += (double)th[i];
        s[1] += (double)qv[i];
    }
    block_sum(s, sh);
    if (threadIdx.x == 0) {
        double n = (double)(d.nx - 2.);
        double tb = s[0] / n, qb = s[1] / n;
        if (a.ref_th) { tb += a.ref_th[k]; qb += a.ref_qv[k]; }
        double tv = tb * (1 + 0.608 * qb);
        a.thb[k] = tb;
        a.qvb[k] = qb;
        a.thvb[k] = tv;
        if (k == 1) { a.thb[0] = tb; a.qvb[0] = qb; a.thvb[0] = tv; }
        if (k == d.nz - 2) { a.thb[d.nz - 1] = tb; a.qvb[d.nz - 1] = qb; a.thvb[d.nz - 1] = tv; }
        if (k == 1 && a.rotate_ubar) a.ubar[0] = a.ubar[1];
    }
}
template <typename T>
__global__ void k_update_mean(MeanArgs<T> a) { k_update_mean_body<T>(a); }

// ---------------------------------------------------------------------------
// cal_u (PoissonSolver.cpp:580-653): the top-row wind from the periodic chi
// problem and the column integral below it.
//
// Top row: chi[i-1] - 2 chi[i] + chi[i+1] = h[i] only enters through
// uxi = (chi[i] - chi[i-1])/dx with its mean removed. The differences satisfy
// d[i+1] - d[i] = h[i], so uxi is an exclusive prefix sum of h (any constant
// cancels in the mean removal); the reference reaches the same values with
// CG to 1e-12. Every block of the column kernel computes the whole top row
// (one block's worth of work, the same arithmetic in every block) and keeps
// its own 32 columns: no second launch waits for a one-block kernel.

template <typename T>
struct CalUArgs {
    Dims d;
    Consts c;
    Profiles p;
    T* u;
    const T *w, *zetap;
    const double* ubar;   // [1] = ubarTopp
};

constexpr int kCalUThreads = 1024;

// The top-row u of columns own_lo .. own_lo+31 into own[] (kCalUThreads
// threads, one block).
template <typename T>
__device__ __forceinline__ void cal_u_top_row(const CalUArgs<T>& a, T* own, int own_lo) {
    __shared__ double sh[32 * 1];
    __shared__ double scan[32];
    const Dims& d = a.d;
    const int NX = d.nx - 2, t = d.nz - 2;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = (NX + kCalUThreads - 1) / kCalUThreads;
    const int i0 = 1 + tid * per;
    const double c = a.p.rhow[t] / a.p.rhou[t];
    double h[kGSMaxPerThread];
    double s[1] = {0};
#pragma unroll
    for (int e = 0; e < kGSMaxPerThread; e++) {
        int i = i0 + e;
        h[e] = 0;
        if (e < per && i <= NX) {
            h[e] = -(0. - a.p.rhow[t] * (double)a.w[d.at(i, t)]) / a.p.rhou[t] * a.c.dx * a.p.hfac;
            s[0] += h[e];
        }
    }
    (void)c;
    block_sum(s, sh);
    const double hmean = s[0] / NX;
    double loc = 0;
#pragma unroll
    for (int e = 0; e < kGSMaxPerThread; e++) {
        int i = i0 + e;
        if (e < per && i <= NX) { h[e] = h[e] - hmean; loc += h[e]; }
    }
    // exclusive scan of the chunk totals
    double incl = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        double p = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += p;
    }
    if (lane == 31) scan[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        double x = scan[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            double p = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += p;
        }
        scan[lane] = x;
    }
    __syncthreads();
    double run = incl - loc + (wid > 0 ? scan[wid - 1] : 0.0);
    double ux[kGSMaxPerThread];
    double s2[1] = {0};
#pragma unroll
    for (int e = 0; e < kGSMaxPerThread; e++) {
        int i = i0 + e;
        ux[e] = 0;
        if (e < per && i <= NX) {
            ux[e] = run * a.c.rdx;
            run += h[e];
            s2[0] += ux[e];
        }
    }
    block_sum(s2, sh);
    const double umean = s2[0] / NX;
    const double ubarp = a.ubar[1];
#pragma unroll
    for (int e = 0; e < kGSMaxPerThread; e++) {
        int i = i0 + e;
        if (e < per && i <= NX && i >= own_lo && i < own_lo + 32) own[i - own_lo] = T((ux[e] - umean) + ubarp);
    }
}

// Column integral u(i, k) = u(i, nz-2) + sum_{m=k}^{nz-3} (dw/dx - rhow zeta)(-dz)
// from the top down (PoissonSolver.cpp:644-651), with the center halo of u;
// u(i, nz-2), the top row, comes from cal_u_top_row in the same block.
// A block owns 32 columns (lanes) and kColSeg z-segments (warps): each thread
// sums its segment, the segment totals are scanned from the top in shared
// memory, then each thread writes its rows. Thirty-two segments give the 64
// blocks of a 2048-column grid 32 warps each (about 8 rows a thread at
// NZ = 256), so the short chains, not a few long ones, set the time.
constexpr int kColSeg = 32;

template <typename T>
__device__ __forceinline__ void k_cal_u_columns_body(const CalUArgs<T>& a) {
    static_assert(32 * kColSeg == kCalUThreads, "the top row takes the column kernel's block");
    __shared__ T tot[kColSeg][32];
    __shared__ T utop_sh[32];
    const Dims& d = a.d;
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    const int i = 1 + blockIdx.x * 32 + lane;
    const bool act = (i <= d.nx - 2);
    const int t = d.nz - 2, nrow = d.nz - 3;               // rows k = 1..nz-3
    // segment s covers rows from the top: k in (khi - len, khi]
    const int r0 = (s * nrow) / kColSeg, r1 = ((s + 1) * nrow) / kColSeg;
    const T rdx = T(a.c.rdx);
    auto term = [&](int k) -> T {
        return ((a.w[d.at(i, k + 1)] - a.w[d.at(i - 1, k + 1)]) * rdx - T(a.p.rhow[k + 1]) * a.zetap[d.at(i, k + 1)]) *
               T(-a.p.dzw[k + 1]);
    };
    cal_u_top_row(a, utop_sh, 1 + blockIdx.x * 32);
    T sum = T(0);
    if (act)
        for (int r = r0; r < r1; r++) sum += term(t - 1 - r);
    tot[s][lane] = sum;
    __syncthreads();
    if (!act) return;
    const T utop = utop_sh[lane];
    T area = T(0);
    for (int q = 0; q < s; q++) area += tot[q][lane];
    if (s == 0) store_center(a.u, d, i, t, utop);
    for (int r = r0; r < r1; r++) {
        int k = t - 1 - r;
        area += term(k);
        store_center(a.u, d, i, k, area + utop);
    }
}
template <typename T>
__global__ void __launch_bounds__(32 * kColSeg) k_cal_u_columns(CalUArgs<T> a) { k_cal_u_columns_body<T>(a); }

}  // namespace vvm
