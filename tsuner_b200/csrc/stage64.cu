// stage64.cu -- FP64 plain form: one fused kernel per RK stage.
//
// Replaces the reference chain reconstructor (GPU/Reconstructor.cu:90) ->
// VolumeSolver (GPU/VolumeSolver.cu:217) -> states_updater
// (GPU/Volume_kernel.cu:180) and, on the last stage of a step, also
// hmax/bmin/eta_max_calculator (GPU/Volume_kernel.cu:79-110), GetDeltaT
// (:19-43) and MinReduction (GPU/Reduction_kernel_min.cu:155-196).
//
// A CTA owns a TX x TY tile of cells.  Phases, separated by __syncthreads():
//   1. stage state (5 planes) + mask of the tile and a 2-cell halo -> smem
//      (halo indices clamped -- which reproduces the reference's im/ip/jm/jp
//      clamping -- or wrapped for periodic boundaries);
//   2. per-cell velocity and concentration, once per cell;
//   3. MUSCL faces (x: L/R, y: D/U) of the tile plus one halo cell per side,
//      positivity-filtered, and the hydrostatic slopes for the source term;
//   4. every edge of the tile evaluated once (boundary ghosts / CC series /
//      periodic seam as in GPU/VolumeSolver.cu:217-408) -> fluctuations;
//   5. per cell: pressure source, friction, erosion/deposition, flux
//      divergence, RK combine, positivity filter, store; on the last stage
//      also the running extrema and the CFL dt partial, with the global
//      minimum finished by the last CTA to arrive (no host round trip).
// Face states and fluxes never touch global memory: per cell-step the
// kernel moves the 250 algorithmic bytes instead of the reference's ~2 KB.
// Phases 3 and 4 each have a single call site of the reconstruction and of
// the Riemann solver (boundary cases only select operands), which keeps the
// kernel body small enough for the instruction cache.
// What bounds it: the dependent FP64 instructions of ~50 divisions and ~20
// roots per cell and stage.  They are evaluated without branches and with
// shared reciprocals (ieee64.h), each phase with one test that sends the
// operands it cannot take to a general form of the same formulas.  4096^2,
// the N-wave entering still water, 2 steps: 12.1 -> 8.9 ms; 1021 x 773 with
// currents everywhere, 4 steps: 1356 -> 900 us (FP64 pipe 34 -> 50 % busy, 117
// -> 88 warp instructions per cell in the first stage, 60 % issue).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

#include "physics64.cuh"
#include "async.cuh"
#include "stage64.h"

namespace tsu {

// A TX x TY tile processed by NTHR threads (NTHR >= TX*TY: the first TX*TY
// threads own a cell in the update; all of them share the halo loads, faces
// and edges).
template <int TX_, int TY_, int NTHR_ = TX_ * TY_>
struct Tile {
    static constexpr int TX = TX_, TY = TY_, NT = NTHR_;
    static constexpr bool kSmall = TX * TY <= 64;  // the small grids' tile
    static_assert(NTHR_ >= TX_ * TY_ && NTHR_ % 32 == 0 && NTHR_ <= 1024, "threads per tile");
    static constexpr int LX = TX + 4, LY = TY + 4, PS = LX * LY;  // loaded tile, 2-cell halo
    static constexpr int FXW = TX + 2, FYH = TY + 2;               // faces incl. one halo cell
    static constexpr int kSV = 5 * PS, kSUC = 3 * PS, kFlux = 20 * TY * TX;
    static constexpr int kRegA = (kSV + kSUC) > kFlux ? (kSV + kSUC) : kFlux;
    static constexpr int kFx = 10 * TY * FXW, kFy = 10 * FYH * TX, kDeta = 2 * TY * TX, kRed = NT / 32;
    static constexpr int kSeam = 4 * (TX + TY);  // seam discharges (periodic grids with a boundary series)
    static constexpr int kDoubles = kRegA + kFx + kFy + kDeta + kRed + kSeam;
    // the 1-byte mask: rows of MLX = TX + 32 cells starting 16 left of the
    // tile (a 16-byte aligned TMA origin for bytes), 128-byte aligned
    static constexpr int MHX = 16, MLX = TX + 2 * MHX, MPS = MLX * LY;
    static constexpr size_t kMaskOff = (sizeof(double) * kDoubles + 127) / 128 * 128;
    // the owned cells' U^n (5 planes) and running extrema (3 planes), [8][TY][TX],
    // staged by TMA in the second RK stage (OWN == 2), 128-byte aligned
    static constexpr size_t kOwnOff = (kMaskOff + MPS + 127) / 128 * 128;
    static constexpr size_t kOwnBytes = 8 * TX * TY * sizeof(double);
    // + 128: the base is rounded up to 128 bytes (TMA destination)
    static constexpr size_t smem(bool staged_own = false) {
        return (staged_own ? kOwnOff + kOwnBytes : kMaskOff + MPS + 16) + 128;
    }
};

__device__ __forceinline__ int wrap_clamp(int g, int n, bool periodic) {
    if (periodic) {
        g %= n;
        return g < 0 ? g + n : g;
    }
    return g < 0 ? 0 : (g >= n ? n - 1 : g);
}

// MUSCL reconstruction of one cell along one direction, GPU/Reconstructor.cu
// :124-194 (x) / :207-271 (y).  c/l/r index the centre and its two
// neighbours in the smem tile (plane stride PS).  Returns the two faces
// (minus side, plus side) before the state filter and the hydrostatic slope
// deta; `ok` as in physics64.cuh.
template <int PS, bool FAST>
__device__ __forceinline__ void reconstruct_dir(const double *sV, const double *sUC, int c, int l, int r,
                                                State5 &fm, State5 &fp, double &deta, bool &ok) {
    const double hi = sV[c], Hi = sV[3 * PS + c];
    const double hl = sV[l], Hl = sV[3 * PS + l];
    const double hr = sV[r], Hr = sV[3 * PS + r];
    const double ci = sUC[2 * PS + c], cl = sUC[2 * PS + l], cr = sUC[2 * PS + r];
    const double uix = sUC[c], uiy = sUC[PS + c];
    const double ulx = sUC[l], uly = sUC[PS + l];
    const double urx = sUC[r], ury = sUC[PS + r];

    double dl = hi - hl, dr = hr - hi;
    double dh = limit<FAST>(dl, dr, ok);
    if (0.5 * fabs(dh) > hi) dh = 2.0 * hi * sgn(dh);
    fm.h = hi - 0.5 * dh;
    fp.h = hi + 0.5 * dh;

    // pos(x) = fmax(x, 0)
    auto pos = [](double x) { return (x > 0.0) ? x : 0.0; };
    double zm = fmin(Hl, Hi);
    dl = pos(hi - Hi + zm) - pos(hl - Hl + zm);
    zm = fmin(Hr, Hi);
    dr = pos(hr - Hr + zm) - pos(hi - Hi + zm);
    deta = limit<FAST>(dl, dr, ok);
    double dz = dh - deta;
    fm.H = Hi - 0.5 * dz;
    fp.H = Hi + 0.5 * dz;

    const double qxi = sV[PS + c], qyi = sV[2 * PS + c];
    dl = uix - ulx;
    dr = urx - uix;
    double du = limit<FAST>(dl, dr, ok);
    double dq = hi * du + uix * dh;
    fm.qx = qxi - 0.5 * dq;
    fp.qx = qxi + 0.5 * dq;
    dl = uiy - uly;
    dr = ury - uiy;
    du = limit<FAST>(dl, dr, ok);
    dq = hi * du + uiy * dh;
    fm.qy = qyi - 0.5 * dq;
    fp.qy = qyi + 0.5 * dq;

    dl = ci - cl;
    dr = cr - ci;
    du = limit<FAST>(dl, dr, ok);
    fm.hc = (ci - 0.5 * du) * fm.h;
    fp.hc = (ci + 0.5 * du) * fp.h;
}

__device__ __forceinline__ void put5(double *base, int stride, const Face5 &s) {
    base[0] = s.h;
    base[stride] = s.u;
    base[2 * stride] = s.v;
    base[3 * stride] = s.H;
    base[4 * stride] = s.c;
}
__device__ __forceinline__ Face5 get5(const double *base, int stride) {
    Face5 s;
    s.h = base[0];
    s.u = base[stride];
    s.v = base[2 * stride];
    s.H = base[3 * stride];
    s.c = base[4 * stride];
    return s;
}
// A face in the frame of the normal (0, 1): velocity along it and along it
// turned left (GPU/VolumeSolver.cu:24-27).  Faces along y are kept this way.
__device__ __forceinline__ Face5 to_y(const Face5 &f) {
    Face5 r = f;
    r.u = f.v;
    r.v = -f.u;
    return r;
}
template <bool FAST, bool FRONT = false>
__device__ __forceinline__ Face5 filtered(State5 &s, bool &ok) {
    if (FRONT) return filter_near_front(s.h, s.qx, s.qy, s.H, s.hc, ok);
    return filter_face<FAST>(s.h, s.qx, s.qy, s.H, s.hc, ok);
}

// Both faces of a cell along one direction, filtered, to shared memory.
// False (FAST only): an operand was out of range and what was stored is not
// valid.  qplus / qminus (may be null): the discharges of the plus-side face
// normal to its edge and of the minus-side face along it, for the periodic
// seam (ydir: the direction is y).
template <int PS, bool FAST, bool FRONT = false>
__device__ __forceinline__ bool make_faces(const double *sV, const double *sUC, int c, int step, double *dst,
                                           int fstride, int side, double *deta_out, double *qplus = nullptr,
                                           double *qminus = nullptr) {
    bool ok = true;
    State5 m, p;
    double deta;
    reconstruct_dir<PS, FAST>(sV, sUC, c, c - step, c + step, m, p, deta, ok);
    Face5 fm = filtered<FAST, FRONT>(m, ok), fp = filtered<FAST, FRONT>(p, ok);  // GPU/Reconstructor.cu:344-348
    if (step != 1) {
        fm = to_y(fm);
        fp = to_y(fp);
    }
    put5(dst, fstride, fm);
    put5(dst + side, fstride, fp);
    if (deta_out) *deta_out = deta;
    if (qplus) *qplus = (step != 1) ? p.qy : p.qx;
    if (qminus) *qminus = (step != 1) ? m.qx : m.qy;
    return ok;
}
// FRONT: the near_front form first (not for a wide tile).  It pays on the small
// grids' tile, where one face by the ordinary operators sets the time of the
// stage (48 x 36 cells with a coast: 23.0 -> 19.7 us per step), and on a tile
// full of such faces (1021 x 773, every cell at 8.5 m/s: 400 -> 338); the large
// tile's warps hide a few of them, and there it cost 2 %.
template <int PS, bool FRONT>
__device__ __noinline__ void make_faces_any(const double *sV, const double *sUC, int c, int step, double *dst,
                                            int fstride, int side, double *deta_out, double *qplus, double *qminus,
                                            bool wide) {
    if (FRONT && !wide &&
        make_faces<PS, true, true>(sV, sUC, c, step, dst, fstride, side, deta_out, qplus, qminus))
        return;
    make_faces<PS, false>(sV, sUC, c, step, dst, fstride, side, deta_out, qplus, qminus);
}

// The fluctuations of one edge, in its frame, to the cells on its two sides
// (null: the side is not in the tile).
template <bool FAST>
__device__ __forceinline__ bool put_edge(const Phys64 &P, const Face5 &a, const Face5 &b, int fixed, double *outM,
                                         double *outP, int FS) {
    double Dm[5], Dp[5];
    const bool ok = edge_flux<FAST>(P, a, b, fixed, Dm, Dp);
#pragma unroll
    for (int f = 0; f < 5; f++) {
        if (outM) outM[f * FS] = Dm[f];
        if (outP) outP[f * FS] = Dp[f];
    }
    return ok;
}
__device__ __noinline__ void put_edge_any(const Phys64 &P, Face5 a, Face5 b, int fixed, double *outM, double *outP,
                                          int FS) {
    put_edge<false>(P, a, b, fixed, outM, outP, FS);
}

// Friction (GPU/Reconstructor.cu:33-55) on the momentum (k1, k2) and the
// erosion/deposition rate phi (:57-88), from U^n = v0; one velocity
// evaluation serves both.  Divisors: h + EPSILON (2^-52 .. 2^100), h + eps_h
// and vs (bounded by plain_sources), 1 + cf with cf < 2^132, 1 + 4.3e-7 Z^5.
template <bool FAST, bool FRONT = false>
__device__ __forceinline__ bool sources(const Phys64 &P, double dt, const double v0[5], double &k1, double &k2,
                                        double &phi) {
    bool ok = true;
    double ux, uy, modu;
    const Divisor<FAST> d0(v0[0] + kEpsilon, ok);
    if constexpr (FAST) {
        if constexpr (FRONT) {
            Divisor<true> dv = d0;
            velocity_near_front(v0[0], v0[1], v0[2], dv, ux, uy, ok);
        } else {
            ux = d0.of(v0[1]);
            uy = d0.of(v0[2]);
        }
        const double m2 = ux * ux + uy * uy;
        // an empty cell: every quotient by EPSILON or eps_h is a zero
        if constexpr (FRONT) ok &= mid_or_zero(m2) & mid(v0[0] + P.eps_h);
        else
            ok &= (wet_divisor(d0.d) & calm(v0[1], ux) & calm(v0[2], uy) & mid_or_zero(m2)) |
                  (empty(v0[0], v0[1], v0[2], v0[4]) & mid(P.eps_h));
        modu = root(m2);
    } else {
        velocity(v0[0], v0[1], v0[2], ux, uy);
        modu = dsqrt(ux * ux + uy * uy);
    }
    if (!FAST && P.manning) {  // GPU/Reconstructor.cu:47-50 as written (multiplies)
        const double cm = dt * P.FR * P.FR * modu / pow(v0[0], 4.0 / 3.0);
        k1 *= cm;
        k2 *= cm;
    } else {
        const double f = dt * P.FR * modu;
        if (FAST) ok &= small_or_zero(f);
        const double cf = d0.of(f);
        const Divisor<FAST> d1(1.0 + cf, ok);
        k1 = d1.of(k1, ok);
        k2 = d1.of(k2, ok);
    }
    const double c = Divisor<FAST>(v0[0] + P.eps_h, ok).of(v0[4], ok);
    const double A = P.k.A_er * (modu * P.k.sqrt_FR);
    double Z;
    if (FAST) {
        ok &= mid_or_zero(A);
        Z = quot(A, P.k.vs, P.inv_vs);
    } else {
        Z = ddiv(A, P.k.vs);
    }
    const double Z5 = Z * Z * Z * Z * Z;
    const double Es = Divisor<FAST>(1 + 4.3e-7 * Z5, ok).of(1.3e-7 * Z5, ok);
    double Fe = P.k.VP * Es;
    if (Fe > 0.1) Fe = 0.1;
    Fe = Fe * (double)(Fe > 0.0);
    double Cb = P.k.K_dep * c;
    double Fd = P.k.vs * Cb;
    if (Fd > 0.1) Fd = 0.1;
    Fd = Fd * (double)(Fd > 0.0);
    phi = (Fe - Fd) * (double)P.suspension;
    return ok;
}
struct Sources {
    double k1, k2, phi;
};
template <bool FRONT>
__device__ __noinline__ Sources sources_any(const Phys64 &P, double dt, State5 v, double k1, double k2) {
    const double v0[5] = {v.h, v.qx, v.qy, v.H, v.hc};
    Sources r;
    r.k1 = k1;
    r.k2 = k2;
    if (FRONT && !P.plain_sources && sources<true, true>(P, dt, v0, r.k1, r.k2, r.phi)) return r;
    r.k1 = k1;
    r.k2 = k2;
    sources<false>(P, dt, v0, r.k1, r.k2, r.phi);
    return r;
}

// RK0: MUSCL-Hancock (RK == 0 of the reference): one stage per step
// (FIRST = LAST = true), the state ping-pongs between bufA and bufB like the
// order-1 form, and bufK holds the unfiltered working state Vk that the
// reference carries from step to step (GPU/Volume_kernel.cu:283-299).
// OWN: where the second RK stage keeps U^n of the owned cell and its running
// extrema between tile start and the update.  0: U^n loaded into registers
// at tile start (held through the face and edge phases), extrema loaded in
// the update; 1: both requested into L2 at tile start and loaded in the
// update; 2: interior tiles stage both into shared memory with TMA boxes
// issued at tile start (they land during the face and edge phases), other
// tiles as 1.
template <int TX, int TY, int NTHR, int MINB, int ORDER, bool FIRST, bool LAST, bool RK0 = false, int OWN = 0>
__global__ void __launch_bounds__(NTHR, MINB) stage64_kernel(const __grid_constant__ Stage64Args A) {
    static_assert(!RK0 || (FIRST && LAST), "MUSCL-Hancock is a single stage");
    constexpr bool PINGPONG = (ORDER == 1) || RK0;
    constexpr bool LATE = (OWN >= 1);
    using T = Tile<TX, TY, NTHR>;
    constexpr int NT = T::NT, LX = T::LX, PS = T::PS, FXW = T::FXW, FYH = T::FYH;
    constexpr int MHX = T::MHX, MLX = T::MLX;
    extern __shared__ __align__(16) double smem_raw[];
    double *smem = smem_align<128>(smem_raw);
    __shared__ uint64_t sBar;     // the tile's TMA load
    __shared__ uint64_t sBarOwn;  // OWN == 2: the owned cells' U^n and extrema
    // cells of the tile and its halo that need the general form, and kWide for
    // each that is not limited()
    __shared__ int sOdd;
    constexpr int kWide = 1 << 16;
    const Phys64 &P = A.phys;
    double *sV = smem;                  // [5][LY][LX]
    double *sUC = smem + T::kSV;        // [3][LY][LX]  (ux, uy, c)
    double *sFlux = smem;               // [4][5][TY][TX]  aliases sV/sUC (dead by then)
    double *sFx = smem + T::kRegA;      // [2][5][TY][FXW]
    double *sFy = sFx + T::kFx;         // [2][5][FYH][TX]
    double *sDeta = sFy + T::kFy;       // [2][TY][TX]
    double *sRed = sDeta + T::kDeta;    // [NT/32]
    double *sSeam = sRed + T::kRed;     // [2][2 TY + 2 TX]
    unsigned char *sM = reinterpret_cast<unsigned char *>(smem) + T::kMaskOff;  // [LY][MLX], tile at column MHX
    __shared__ int sLast;

    const int npx = P.npx, npy = P.npy;
    const bool periodic = (P.wbc == 2);
    const int tid = threadIdx.x;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const long long pitch = A.pitch, plane = A.plane;

    if (threadIdx.x == 0) {  // barriers of the tile's loads, before anything the previous kernel may still hold up
        mbar_init(&sBar, 1);
        if (OWN == 2 && !FIRST) mbar_init(&sBarOwn, 1);
        mbar_init_fence();
        sOdd = 0;
    }
    prior_grids_done();
    next_grid_may_start();

    const double *Vin;
    const double *V0;
    double *Vout;
    int par = 0;
    if (!PINGPONG) {
        Vin = FIRST ? A.bufA : A.bufB;
        V0 = A.bufA;
        Vout = FIRST ? A.bufB : A.bufA;
    } else {
        par = (int)A.scal[SC_PAR];
        Vin = par ? A.bufB : A.bufA;
        V0 = Vin;
        Vout = par ? A.bufA : A.bufB;
    }

    // tile and halo inside the stored rows (the owned rows and a slab's ghost
    // rows), not periodic: no clamping, and every edge of the tile is an
    // interior edge
    const bool inner =
        !periodic && x0 >= 2 && y0 - 2 >= -P.gs && x0 + TX + 2 <= npx && y0 + TY + 2 <= npy + P.gn;

    // ---- phase 1: tile + halo -> smem.  Interior tiles: one TMA box of the
    // 5 state planes (x0 - 2 doubles = a multiple of 16 bytes) and one of the
    // mask (from x0 - 16); boundary tiles (clamped or wrapped halo) with
    // ordinary loads.
    const bool use_tma = inner && A.tma;
    // the owned cells of an interior tile lie inside the stored rows: the
    // boxes at (x0, y0) are in bounds, x0 * 8 bytes a multiple of 256
    const bool own_tma = (OWN == 2) && !FIRST && use_tma;
    constexpr int TC = TX * TY;
    double *sOwn = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(smem) + T::kOwnOff);
    if (use_tma) {
        if (tid == 0) {
            mbar_expect_tx(&sBar, 5 * PS * sizeof(double) + T::MPS);
            // the tensor maps start at the first stored row (a slab's lowest ghost row)
            tma_load_3d(sV, (Vin == A.bufB) ? &A.tmB : &A.tmA, x0 - 2, y0 - 2 + P.gs, 0, &sBar);
            tma_load_2d(sM, &A.tmM, x0 - MHX, y0 - 2 + P.gs, &sBar);
            if (own_tma) {
                mbar_expect_tx(&sBarOwn, (LAST ? 8 : 5) * TC * sizeof(double));
                tma_load_3d(sOwn, &A.tmO, x0, y0 + P.gs, 0, &sBarOwn);
                if (LAST) {
#pragma unroll
                    for (int f = 0; f < 3; f++) tma_load_2d(sOwn + (5 + f) * TC, &A.tmE[f], x0, y0 + P.gs, &sBarOwn);
                }
            }
        }
    } else {
        for (int idx = tid; idx < PS; idx += NT) {
            const int ly = idx / LX, lx = idx - ly * LX;
            int gx = x0 + lx - 2, gy = y0 + ly - 2;
            if (!inner) {
                gx = wrap_clamp(gx, npx, periodic);
                // rows outside the stored ones: the grid's own boundary (a
                // slab stores ghost rows wherever it has a neighbour)
                if (gy < -P.gs || gy >= npy + P.gn) gy = wrap_clamp(gy, npy, periodic);
            }
            const long long g = (long long)gy * pitch + gx;
#pragma unroll
            for (int f = 0; f < 5; f++) sV[f * PS + idx] = Vin[f * plane + g];
            sM[ly * MLX + lx + (MHX - 2)] = A.mask[g];
        }
    }
    const bool cell_thread = tid < TX * TY;  // owns a cell in the update
    const int tx = cell_thread ? tid % TX : 0, ty = cell_thread ? tid / TX : 0;
    const int gi = x0 + tx, gj = y0 + ty;
    const bool own = cell_thread && (gi < npx) && (gj < npy);
    const long long gown = (long long)(own ? gj : 0) * pitch + (own ? gi : 0);
    double v0[5];
    if (!FIRST && !own_tma) {  // U^n of the owned cell (friction, erosion, RK combine)
#pragma unroll
        for (int f = 0; f < 5; f++) {
            if (LATE) prefetch_l2(V0 + f * plane + gown);
            else v0[f] = V0[f * plane + gown];
        }
    }
    if (LATE && LAST && own && !own_tma) {
        prefetch_l2(A.hmax + gown);
        prefetch_l2(A.bmin + gown);
        prefetch_l2(A.eta_max + gown);
    }
    // the scalars are read while the boxes travel
    const double t = A.scal[SC_T], tend = A.scal[SC_TEND], dt = A.scal[SC_DT];
    __syncthreads();
    if (use_tma) {  // every thread sees the box land (bounded wait)
        const bool ok = mbar_wait_first(&sBar, 0);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                A.scal[SC_ERR] = 1.0;
                mbar_wait(&sBar, 0);
                if (own_tma) mbar_wait(&sBarOwn, 0);
            }
            return;
        }
    }

    if (!(t < tend)) {  // run_until predicate (uniform); the other boxes land first
        if (own_tma && tid == 0) mbar_wait(&sBarOwn, 0);
        return;
    }

    const int cidx = (ty + 2) * LX + (tx + 2);
    double vc[5];
#pragma unroll
    for (int f = 0; f < 5; f++) vc[f] = sV[f * PS + cidx];
    if (FIRST) {
#pragma unroll
        for (int f = 0; f < 5; f++) v0[f] = vc[f];
    }

    // ---- phase 2: per-cell velocity and concentration
    int odd = 0;
    for (int idx = tid; idx < PS; idx += NT) {
        const double h = sV[idx], qx = sV[PS + idx], qy = sV[2 * PS + idx], hc = sV[4 * PS + idx];
        bool ok = true;
        Face5 f = face_of<true>(h, qx, qy, 0.0, hc, ok);
        if (!ok) {
            f = face_of<false>(h, qx, qy, 0.0, hc, ok);
            odd += (limited(h) & limited(f.u) & limited(f.v) & limited(f.c)) ? 1 : kWide;
        }
        sUC[idx] = f.u;
        sUC[PS + idx] = f.v;
        sUC[2 * PS + idx] = f.c;
    }
    if (odd) atomicAdd(&sOdd, odd);
    __syncthreads();
    // A tile most of whose cells the branch-free form of the faces refuses
    // (films, speeds from 7 m/s) does not try it first.  1021 x 773, every cell
    // at 8.5 m/s: 459 -> 338 us per step, films of 3e-7 m: 380 -> 290; the same
    // test for the sources and the update gave 4 % more there, but cost every
    // other grid 0.4 %.  Fast cells one by one among calm ones (10 % of them: 477
    // us) would gain from a lower line, 416 at PS / 32 and 379 at PS / 128, but
    // the coast's tiles do not: 4096^2 8.87 -> 8.91 ms for two steps.
    constexpr int kMost = PS / 2;

    // Periodic grids with an expired boundary series mirror the discharge of the
    // seam's low-side face into its high-side face (phase 4).  The faces do not
    // hold discharges, so those of the edges at the grid's two ends are kept
    // aside: which = 0 the low-side face's normal discharge, 1 the high-side
    // face's transverse one; k: row or column of the tile; e: global edge index.
    const bool seam_q = periodic && P.read_files;
    auto seam_slot = [&](bool vert, int which, int k, int e) -> double * {
        const int end = vert ? npx : P.ny_glob;
        if (e != 0 && e != end) return nullptr;
        return sSeam + which * T::kSeam / 2 + (vert ? 0 : 2 * TY) + (e == 0 ? 0 : (vert ? TY : TX)) + k;
    };

    // ---- phase 3: faces (one reconstruction call site)
    if (RK0 && ORDER == 2) {
        // MUSCL-Hancock: the predictor needs all four faces of a cell, so an
        // item is a cell -- the tile, then its halo columns -1 / TX (x faces
        // kept) and halo rows -1 / TY (y faces kept)
        constexpr int NC = TX * TY + 2 * TY + 2 * TX;
        for (int item = tid; item < NC; item += NT) {
            int lx, ly;
            if (item < TX * TY) {
                ly = item / TX;
                lx = item - ly * TX;
            } else if (item < TX * TY + 2 * TY) {
                const int k = item - TX * TY;
                ly = k >> 1;
                lx = (k & 1) ? TX : -1;
            } else {
                const int k = item - TX * TY - 2 * TY;
                lx = k >> 1;
                ly = (k & 1) ? TY : -1;
            }
            const int c = (ly + 2) * LX + (lx + 2);
            State5 L, R, D, U;
            double detx, dety;
            bool ok = true;
            reconstruct_dir<PS, false>(sV, sUC, c, c - 1, c + 1, L, R, detx, ok);
            reconstruct_dir<PS, false>(sV, sUC, c, c - LX, c + LX, D, U, dety, ok);
            hancock_predictor(P, dt, sV[c], detx, dety, L, R, D, U);
            if (ly >= 0 && ly < TY) {
                double *dst = sFx + ly * FXW + (lx + 1);
                put5(dst, TY * FXW, filtered<false>(L, ok));
                put5(dst + 5 * TY * FXW, TY * FXW, filtered<false>(R, ok));
                if (seam_q) {
                    if (double *q = seam_slot(true, 0, ly, x0 + lx + 1)) *q = R.qx;
                    if (double *q = seam_slot(true, 1, ly, x0 + lx)) *q = L.qy;
                }
            }
            if (lx >= 0 && lx < TX) {
                double *dst = sFy + (ly + 1) * TX + lx;
                put5(dst, FYH * TX, to_y(filtered<false>(D, ok)));
                put5(dst + 5 * FYH * TX, FYH * TX, to_y(filtered<false>(U, ok)));
                if (seam_q) {
                    if (double *q = seam_slot(false, 0, lx, P.j0 + y0 + ly + 1)) *q = U.qy;
                    if (double *q = seam_slot(false, 1, lx, P.j0 + y0 + ly)) *q = D.qx;
                }
            }
            if (lx >= 0 && lx < TX && ly >= 0 && ly < TY) {
                sDeta[ly * TX + lx] = detx;
                sDeta[TY * TX + ly * TX + lx] = dety;
            }
        }
    }
    // Otherwise a warp's item is 32 faces: the x faces of RPW tile rows, the y
    // faces of RPW rows (one halo row on each side included), or part of the x
    // faces of the halo columns (two per row), last because it is not full.
    // 19 items for 10 warps: two rounds.
    constexpr int RPW = 32 / TX, WX = TY / RPW, WY = (FYH + RPW - 1) / RPW, WF = (2 * TY + 31) / 32;
    static_assert(32 % TX == 0 && TY % RPW == 0, "tile rows per warp");
    const int warp = tid >> 5, lr = (tid & 31) / TX, lc = (tid & 31) % TX;
    // The loop comes twice, with and without what only seams and such tiles need:
    // 4096^2 4195 us per step, 4226 with that in one loop.
    auto faces = [&](const bool G) __attribute__((always_inline)) {
        for (int item = warp; item < ((RK0 && ORDER == 2) ? 0 : WX + WY + WF); item += NT / 32) {
            const bool xi = item < WX || item >= WX + WY;
            int lx, ly;  // the cell, in tile coordinates
            if (item < WX) {
                lx = lc;
                ly = item * RPW + lr;
            } else if (xi) {
                const int k = (item - WX - WY) * 32 + (tid & 31);
                lx = (k & 1) ? TX : -1;
                ly = k >> 1;
                if (ly >= TY) continue;
            } else {
                lx = lc;
                ly = (item - WX) * RPW + lr - 1;
                if (ly > TY) continue;
            }
            const int c = (ly + 2) * LX + (lx + 2), step = xi ? 1 : LX;
            double *dst = xi ? sFx + ly * FXW + (lx + 1) : sFy + (ly + 1) * TX + lx;
            const int fstride = xi ? TY * FXW : FYH * TX, side = 5 * fstride;
            int didx = -1;  // the cell is in the tile
            if (item < WX) didx = ly * TX + lx;
            else if (!xi && ly >= 0 && ly < TY) didx = TY * TX + ly * TX + lx;
            double *qplus = nullptr, *qminus = nullptr;
            if (G && seam_q) {  // the cell's plus face is at the edge after it, its minus face at the edge before
                const int k = xi ? ly : lx, e = xi ? x0 + lx : P.j0 + y0 + ly;
                qplus = seam_slot(xi, 0, k, e + 1);
                qminus = seam_slot(xi, 1, k, e);
            }
            if (ORDER == 2) {
                if (P.dry_skip && sV[c] == 0.0 && sV[c - step] == 0.0 && sV[c + step] == 0.0) {
                    // a dry stencil: every slope is avg(0, 0) = 0, so both
                    // faces are (0, q_i, 0, H_i, 0 * c) before the filter and
                    // (0, 0, 0, H_i, 0) after it (zeros up to their sign), and
                    // deta = 0
                    Face5 f;
                    f.h = f.u = f.v = f.c = 0.0;
                    f.H = sV[3 * PS + c];
                    put5(dst, fstride, f);
                    put5(dst + side, fstride, f);
                    if (didx >= 0) sDeta[didx] = 0.0;
                    if (G && qplus) *qplus = 0.0;
                    if (G && qminus) *qminus = 0.0;
                } else {
                    double *deta = (didx >= 0) ? sDeta + didx : nullptr;
                    if (G)
                        make_faces_any<PS, true>(sV, sUC, c, step, dst, fstride, side, deta, qplus, qminus,
                                                 sOdd >= kWide);
                    else if (!make_faces<PS, true>(sV, sUC, c, step, dst, fstride, side, deta))
                        make_faces_any<PS, T::kSmall>(sV, sUC, c, step, dst, fstride, side, deta, nullptr, nullptr,
                                                      false);
                }
            } else {  // first order: faces are the cell values (GPU/Reconstructor.cu:99-107)
                Face5 f;
                f.h = sV[c];
                f.u = sUC[c];
                f.v = sUC[PS + c];
                f.H = sV[3 * PS + c];
                f.c = sUC[2 * PS + c];
                if (!xi) f = to_y(f);
                put5(dst, fstride, f);
                put5(dst + side, fstride, f);
                if (G && qplus) *qplus = sV[(step == 1 ? 1 : 2) * PS + c];
                if (G && qminus) *qminus = sV[(step == 1 ? 2 : 1) * PS + c];
            }
        }
    };
    const bool general = seam_q || sOdd > kMost;  // no branch-free form of this tile's faces
    if (general) faces(true);
    else faces(false);
    __syncthreads();

    // ---- phase 4: edges (each once per tile, one Riemann call site)
    const bool series_on = !inner && P.read_files && (t < A.tCC[A.timeCC - 2]);
    constexpr int FS = TY * TX;  // flux plane stride; planes FL, FR, FD, FU, each in its edge's frame
    // A warp's item is 32 edges: the east edges of RPW tile rows, the RPW rows
    // of horizontal edges, or west edges of the tile (TY in all), last.
    constexpr int WH = (TY + 1 + RPW - 1) / RPW, WW = (TY + 31) / 32;
    for (int item = warp; item < WX + WH + WW; item += NT / 32) {
        const bool vert = item < WX || item >= WX + WH;
        int r, e, c;  // vertical edge e (0..TX) of row r, or horizontal edge e (0..TY) of column c
        if (item < WX) {
            r = item * RPW + lr;
            e = lc + 1;
            c = 0;
        } else if (vert) {
            r = (item - WX - WH) * 32 + (tid & 31);
            e = c = 0;
            if (r >= TY) continue;
        } else {
            r = 0;
            e = (item - WX) * RPW + lr;
            c = lc;
            if (e > TY) continue;
        }
        Face5 a, b;
        int n = 1, fixed, seg = 0;
        bool bnd = false, seam = false;
        double *outM = nullptr, *outP = nullptr;
        if (inner) {  // interior edges only (uniform per tile): no bounds or boundary cases
            if (vert) {
                a = get5(sFx + (5 * TY + r) * FXW + e, TY * FXW);
                b = get5(sFx + r * FXW + (e + 1), TY * FXW);
                fixed = (int)sM[(r + 2) * MLX + e + 1 + (MHX - 2)] * (int)sM[(r + 2) * MLX + e + 2 + (MHX - 2)];
                if (e >= 1) outM = sFlux + 1 * 5 * FS + r * TX + (e - 1);
                if (e < TX) outP = sFlux + 0 * 5 * FS + r * TX + e;
            } else {
                a = get5(sFy + (5 * FYH + e) * TX + c, FYH * TX);
                b = get5(sFy + (e + 1) * TX + c, FYH * TX);
                fixed = (int)sM[(e + 1) * MLX + c + 2 + (MHX - 2)] * (int)sM[(e + 2) * MLX + c + 2 + (MHX - 2)];
                if (e >= 1) outM = sFlux + 3 * 5 * FS + (e - 1) * TX + c;
                if (e < TY) outP = sFlux + 2 * 5 * FS + e * TX + c;
            }
        } else if (vert) {
            const int ex = x0 + e, ey = y0 + r;
            if (ey >= npy || ex > npx) continue;
            const int ly = r + 2;
            // R face of tile col e-1 is sFx col e; L face of tile col e is col e+1
            const double *Rf = sFx + (5 * TY + r) * FXW + e;
            const double *Lf = sFx + r * FXW + (e + 1);
            const int J = P.j0 + ey;  // the global row (boundary-series segments)
            if (periodic && (ex == 0 || ex == npx)) {  // seam: GPU/VolumeSolver.cu:262-275,289-298
                a = get5(Rf, TY * FXW);
                b = get5(Lf, TY * FXW);
                fixed = sM[ly * MLX + e + 1 + (MHX - 2)];
                seam = true;
                seg = npx + J;
                if (e >= 1) outM = sFlux + 1 * 5 * FS + r * TX + (e - 1);
                if (e < TX) outP = sFlux + 0 * 5 * FS + r * TX + e;
            } else if (ex == 0) {  // west: GPU/VolumeSolver.cu:233-258
                a = get5(Lf, TY * FXW);
                n = -1;
                fixed = sM[ly * MLX + e + 2 + (MHX - 2)];
                bnd = true;
                seg = 2 * npx + P.ny_glob + J;
                outM = sFlux + 0 * 5 * FS + r * TX + e;
            } else if (ex == npx) {  // east: GPU/VolumeSolver.cu:276-298
                a = get5(Rf, TY * FXW);
                fixed = sM[ly * MLX + e + 1 + (MHX - 2)];
                bnd = true;
                seg = npx + J;
                outM = sFlux + 1 * 5 * FS + r * TX + (e - 1);
            } else {  // interior: GPU/VolumeSolver.cu:300-314
                a = get5(Rf, TY * FXW);
                b = get5(Lf, TY * FXW);
                fixed = (int)sM[ly * MLX + e + 1 + (MHX - 2)] * (int)sM[ly * MLX + e + 2 + (MHX - 2)];
                if (e >= 1) outM = sFlux + 1 * 5 * FS + r * TX + (e - 1);
                if (e < TX) outP = sFlux + 0 * 5 * FS + r * TX + e;
            }
        } else {
            const int ex = x0 + c, ey = y0 + e;
            if (ex >= npx || ey > npy) continue;
            // U face of tile row e-1 is sFy row e; D face of tile row e is row e+1
            const double *Uf = sFy + (5 * FYH + e) * TX + c;
            const double *Df = sFy + (e + 1) * TX + c;
            // the grid's own south / north boundary (a slab's other edges are
            // interior edges, their far side in the ghost rows)
            const int J = P.j0 + ey;
            const bool south = (J == 0), north = (J == P.ny_glob);
            if (periodic && (south || north)) {  // seam: GPU/VolumeSolver.cu:352-367,378-387
                a = get5(Uf, FYH * TX);
                b = get5(Df, FYH * TX);
                fixed = sM[(e + 1) * MLX + c + 2 + (MHX - 2)];
                seam = true;
                seg = npx + P.ny_glob + ex;
                if (e >= 1) outM = sFlux + 3 * 5 * FS + (e - 1) * TX + c;
                if (e < TY) outP = sFlux + 2 * 5 * FS + e * TX + c;
            } else if (south) {  // south: GPU/VolumeSolver.cu:324-349
                a = get5(Df, FYH * TX);
                n = -1;
                fixed = sM[(e + 2) * MLX + c + 2 + (MHX - 2)];
                bnd = true;
                seg = ex;
                outM = sFlux + 2 * 5 * FS + e * TX + c;
            } else if (north) {  // north: GPU/VolumeSolver.cu:352-387
                a = get5(Uf, FYH * TX);
                fixed = sM[(e + 1) * MLX + c + 2 + (MHX - 2)];
                bnd = true;
                seg = npx + P.ny_glob + ex;
                outM = sFlux + 3 * 5 * FS + (e - 1) * TX + c;
            } else {  // interior: GPU/VolumeSolver.cu:389-403
                a = get5(Uf, FYH * TX);
                b = get5(Df, FYH * TX);
                fixed = (int)sM[(e + 1) * MLX + c + 2 + (MHX - 2)] * (int)sM[(e + 2) * MLX + c + 2 + (MHX - 2)];
                if (e >= 1) outM = sFlux + 3 * 5 * FS + (e - 1) * TX + c;
                if (e < TY) outP = sFlux + 2 * 5 * FS + e * TX + c;
            }
        }
        if (bnd) {  // ghost = copy, wall mirror of the normal momentum
            b = a;
            if (P.wbc == 1) b.u = -a.u;
        }
        if ((bnd || seam) && P.read_files) {  // CC series while active, then wall
            if (series_on) {
                State5 g;
                series_state(A.CC, A.tCC, t, npx, P.ny_glob, seg, g);
                bool ok = true;
                b = face_of<false>(g.h, g.qx, g.qy, g.H, g.hc, ok);
                if (!vert) b = to_y(b);
            } else if (bnd) {
                b.u = -a.u;
            } else {
                // the high-side face with the low-side face's normal discharge
                const int k = vert ? r : c, ge = vert ? x0 + e : P.j0 + y0 + e;
                const double qn = -*seam_slot(vert, 0, k, ge), qt = *seam_slot(vert, 1, k, ge);
                velocity(b.h, vert ? qn : qt, vert ? qt : qn, b.u, b.v);
                if (!vert) b = to_y(b);
            }
        }
        if (P.dry_skip && a.h == 0.0 && b.h == 0.0) {
            // Both faces dry (h == 0 exactly, which also excludes NaN): every
            // velocity, flux and depth is a zero, the hydrostatic depths are
            // max(-H + min(H_a, H_b), 0) = 0, both wave speeds are 0, so all
            // ten fluctuations evaluate to zeros.  They are stored as +0 (the
            // full evaluation can give -0 for some; a zero's sign does not
            // reach any non-zero value of this scheme).  Dry land makes this
            // the common edge of a coastal grid.
#pragma unroll
            for (int f = 0; f < 5; f++) {
                if (outM) outM[f * FS] = 0.0;
                if (outP) outP[f * FS] = 0.0;
            }
            continue;
        }
        if (n < 0) {  // the grid's west and south edges: the normal points out of the grid
            a.u = -a.u;
            a.v = -a.v;
            b.u = -b.u;
            b.v = -b.v;
        }
        if (!put_edge<true>(P, a, b, fixed, outM, outP, FS)) put_edge_any(P, a, b, fixed, outM, outP, FS);
        if (n < 0) {
            outM[FS] = -outM[FS];
            outM[2 * FS] = -outM[2 * FS];
        }
    }
    bool own_ok = true;
    if (own_tma) own_ok = mbar_wait_first(&sBarOwn, 0);  // the owned cells' U^n and extrema (bounded wait)
    if (__syncthreads_or(!own_ok)) {
        if (tid == 0) {
            A.scal[SC_ERR] = 1.0;
            mbar_wait(&sBarOwn, 0);
        }
        return;
    }

    // ---- phase 5: cell update
    double dtcell = CUDART_INF;
    bool bad = false;  // last stage: the new state of the owned cell is not finite
    const int cell = ty * TX + tx;
    if (own) {
        if (LATE && !FIRST) {
#pragma unroll
            for (int f = 0; f < 5; f++) v0[f] = own_tma ? sOwn[f * TC + cell] : V0[f * plane + gown];
        }
        double vk[5];  // the reference's Vk: this stage's input, or MUSCL-Hancock's carried working state
#pragma unroll
        for (int f = 0; f < 5; f++) vk[f] = RK0 ? A.bufK[f * plane + gown] : vc[f];
        if (ORDER == 2) {  // pressure source, GPU/Reconstructor.cu:197,274
            const double dtax = dt * P.inv_dx, dtay = dt * P.inv_dy;
            vk[1] -= dtax * kG * vc[0] * sDeta[ty * TX + tx];
            vk[2] -= dtay * kG * vc[0] * sDeta[TY * TX + ty * TX + tx];
        }
        {  // friction and erosion/deposition from U^n
            double k1 = vk[1], k2 = vk[2], phi;
            if (P.plain_sources || !sources<true>(P, dt, v0, k1, k2, phi)) {
                State5 v;
                v.h = v0[0];
                v.qx = v0[1];
                v.qy = v0[2];
                v.H = v0[3];
                v.hc = v0[4];
                const Sources r = sources_any<T::kSmall>(P, dt, v, vk[1], vk[2]);
                k1 = r.k1;
                k2 = r.k2;
                phi = r.phi;
            }
            vk[1] = k1;
            vk[2] = k2;
            vk[3] -= dt * phi;
            vk[4] += dt * phi;
        }
        // flux divergence, GPU/Volume_kernel.cu:191-195
        const double invx = dt * P.inv_dx, invy = dt * P.inv_dy;
#pragma unroll
        for (int f = 0; f < 5; f++) {
            double FL = sFlux[(0 * 5 + f) * FS + cell], FR = sFlux[(1 * 5 + f) * FS + cell];
            // y fluctuations back to x/y components (GPU/VolumeSolver.cu:129-152)
            const int fy = (f == 1) ? 2 : (f == 2) ? 1 : f;
            double FD = sFlux[(2 * 5 + fy) * FS + cell], FU = sFlux[(3 * 5 + fy) * FS + cell];
            if (f == 1) {
                FD = -FD;
                FU = -FU;
            }
            vk[f] -= invx * (FL + FR) + invy * (FD + FU);
        }
        // RK combine + filter, GPU/Volume_kernel.cu:244-281; MUSCL-Hancock
        // filters Vk itself and keeps the unfiltered Vk (:283-299)
        double h, qx, qy, z, hc;
        if (RK0) {
            h = vk[0];
            qx = vk[1];
            qy = vk[2];
            z = vk[3];
            hc = vk[4];
#pragma unroll
            for (int f = 0; f < 5; f++) A.bufK[f * plane + gown] = vk[f];
        } else {
            const int k = (ORDER == 2 && !FIRST) ? 1 : 0;
            const double coef0 = 0.0 * (double)(k == 0) + 0.5 * (double)(k == 1);
            const double coef1 = 1.0 - coef0;
            h = coef0 * v0[0] + coef1 * vk[0];
            qx = coef0 * v0[1] + coef1 * vk[1];
            qy = coef0 * v0[2] + coef1 * vk[2];
            z = coef0 * v0[3] + coef1 * vk[3];
            hc = coef0 * v0[4] + coef1 * vk[4];
        }
        double d;  // last stage: the new cell's CFL step
        {
            bool ok = true;
            double fh = (h < 0.0) ? 0.0 : h, fx = qx, fy = qy, fc = hc;
            const Face5 f = filter_face<true>(fh, fx, fy, z, fc, ok);
            if (LAST) ok &= cfl_dt_fast(P, f, d);
            if (!ok) {
                fh = h;
                fx = qx;
                fy = qy;
                fc = hc;
                positivity_filter(fh, fx, fy, fc);
                if (LAST) d = cfl_dt(P, fh, fx, fy);
            }
            h = fh;
            qx = fx;
            qy = fy;
            hc = fc;
        }
        Vout[gown] = h;
        Vout[plane + gown] = qx;
        Vout[2 * plane + gown] = qy;
        Vout[3 * plane + gown] = z;
        Vout[4 * plane + gown] = hc;
        if (LAST) {
            const double eps_h = P.eps_h;
            if (own_tma) {
                if (h > eps_h) A.hmax[gown] = fmax(sOwn[5 * TC + cell], h);
                A.bmin[gown] = fmax(sOwn[6 * TC + cell], z);
                if (h > eps_h) A.eta_max[gown] = fmax(sOwn[7 * TC + cell], h - z);
            } else {
                if (h > eps_h) A.hmax[gown] = fmax(A.hmax[gown], h);
                A.bmin[gown] = fmax(A.bmin[gown], z);
                if (h > eps_h) A.eta_max[gown] = fmax(A.eta_max[gown], h - z);
            }
            if (!isnan(d)) dtcell = d;
            bad = !(finite64(h) && finite64(qx) && finite64(qy) && finite64(z) && finite64(hc));
        }
    }

    if (LAST) {
        // a NaN / Inf anywhere in the new state is reported to the host (the
        // values themselves are stored unchanged, as the reference would)
        if (__any_sync(0xffffffffu, bad) && (tid & 31) == 0) A.scal[SC_NAN] = 1.0;
        // CTA minimum with warp shuffles; the last CTA to finish reduces the
        // partials, advances t and publishes the next dt
        // (GPU/main_TSUNER.cu:185,190-192).
        double m = dtcell;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((tid & 31) == 0) sRed[tid >> 5] = m;
        __syncthreads();
        if (tid < 32) {
            m = (tid < T::kRed) ? sRed[tid] : CUDART_INF;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (tid == 0) {
                const unsigned nb = gridDim.x * gridDim.y;
                const unsigned b = blockIdx.y * gridDim.x + blockIdx.x;
                A.partials[b] = m;
                __threadfence();
                unsigned tk = atomicAdd(A.ticket, 1u);
                sLast = (tk == nb - 1);
            }
        }
        __syncthreads();
        if (sLast) {
            __threadfence();
            const unsigned nb = gridDim.x * gridDim.y;
            double mm = CUDART_INF;
            for (unsigned i = tid; i < nb; i += NT) mm = fmin(mm, __ldcg(A.partials + i));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mm = fmin(mm, __shfl_xor_sync(0xffffffffu, mm, o));
            __syncthreads();
            if ((tid & 31) == 0) sRed[tid >> 5] = mm;
            __syncthreads();
            if (tid == 0) {
                for (int w = 0; w < T::kRed; w++) mm = fmin(mm, sRed[w]);
                A.scal[SC_T] = t + dt;
                A.scal[SC_DT] = finalize_dt(mm, (long long)npx * P.ny_glob);
                A.scal[SC_STEPS] += 1.0;
                if (PINGPONG) A.scal[SC_PAR] = (double)(1 - par);
                *A.ticket = 0u;
                __threadfence();
            }
        }
    }
}

// GetDeltaT + MinReduction over a state (initial dt, GPU/main_TSUNER.cu:147-148).
__global__ void __launch_bounds__(256) dt_partials_kernel(const double *__restrict__ V, long long pitch,
                                                          long long plane, Phys64 P, double *partials,
                                                          unsigned *ticket, double *scal) {
    __shared__ double sRed[8];
    __shared__ int sLast;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int gi = blockIdx.x * blockDim.x + threadIdx.x, gj = blockIdx.y * blockDim.y + threadIdx.y;
    double m = CUDART_INF;
    bool bad = false;
    if (gi < P.npx && gj < P.npy) {
        long long g = (long long)gj * pitch + gi;
        double d = cfl_dt(P, V[g], V[plane + g], V[2 * plane + g]);
        if (!isnan(d)) m = d;
        bad = !(finite64(V[g]) && finite64(V[plane + g]) && finite64(V[2 * plane + g]) &&
                finite64(V[3 * plane + g]) && finite64(V[4 * plane + g]));
    }
    if (__any_sync(0xffffffffu, bad) && (tid & 31) == 0) scal[SC_NAN] = 1.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0) sRed[tid >> 5] = m;
    __syncthreads();
    const unsigned nb = gridDim.x * gridDim.y;
    if (tid == 0) {
        for (int w = 1; w < 8; w++) m = fmin(m, sRed[w]);
        partials[blockIdx.y * gridDim.x + blockIdx.x] = m;
        __threadfence();
        sLast = (atomicAdd(ticket, 1u) == nb - 1);
    }
    __syncthreads();
    if (sLast) {
        __threadfence();
        double mm = CUDART_INF;
        for (unsigned i = tid; i < nb; i += 256) mm = fmin(mm, __ldcg(partials + i));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mm = fmin(mm, __shfl_xor_sync(0xffffffffu, mm, o));
        __syncthreads();
        if ((tid & 31) == 0) sRed[tid >> 5] = mm;
        __syncthreads();
        if (tid == 0) {
            for (int w = 0; w < 8; w++) mm = fmin(mm, sRed[w]);
            scal[SC_DT] = finalize_dt(mm, (long long)P.npx * P.ny_glob);
            *ticket = 0u;
            __threadfence();
        }
    }
}

__global__ void fill_kernel(double *p, long long n, double v) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        p[i] = v;
}

// Per-run constants with the reference expressions (device pow()).
__global__ void consts_kernel(SimParams p, TsuConsts *k) {
    double nu = 1.002e-6;
    double s = p.R - 1.0;
    k->vs = sqrt((13.95 * nu / p.DS) * (13.95 * nu / p.DS) + 1.09 * s * kG * p.DS) - 13.95 * nu / p.DS;
    k->Rp = (p.DS * sqrt(s * kG * p.DS)) / nu;
    double a1, a2;
    if (k->Rp > 2.36) {
        a1 = 1;
        a2 = 0.6;
    } else {
        a1 = 0.586;
        a2 = 1.23;
    }
    k->A_er = a1 * pow(k->Rp, a2);
    k->sqrt_FR = sqrt(p.FR);
    k->VP = k->vs * (1 - p.porosity);
    k->K_dep = (1.64 + 0.4 * pow(p.DS / p.Dsg, 1.64));
    k->sqrt_OC = sqrt(p.OC);
    k->DS5 = 5 * p.DS;
}

// ------------------------------------------------------------------ host side
static_assert(kDefaultWaitNs == kWaitNs, "one default wait limit");

cudaError_t set_wait_limit_stage64(unsigned long long ns) {
    return cudaMemcpyToSymbol(g_wait_limit_ns, &ns, sizeof(ns));
}

EncodeTiledFn tensor_map_encoder() {
    static EncodeTiledFn f = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return f;
}

namespace {

// Grids of up to one wave of 16 x 4 tiles (three CTAs on each of 148 SMs) use
// those: a tile is then one round of its warps, and more SMs have work.  Beyond
// it they need a second wave, with 1.5 times the halo cells per owned one, where
// 32 x 8 tiles need one.  On narrow grids, where most 32 x 8 tiles lie at a
// boundary and wait for their few faces of the general form, the second wave
// costs no more until it is two thirds full.  us per step, 16 x 4 against
// 32 x 8, still water entered by a wave / moving water with humps:
//   48 x 36 (27 tiles of 16 x 4)  18.2 / 21.0  26.8 / 31.4
//   384 x 72 (432)                22.7 / 20.7  25.4 / 27.5
//   768 x 44 (528)                34.7 / 27.0  28.9 / 23.5
//   256 x 248 (992)               41.5 / 39.3  32.5 / 36.0
//   128 x 224 (448)               28.5 / 26.9  28.9 / 31.9
//   96 x 440 (660)                34.0 / 31.5  34.4 / 39.6
//   96 x 592 (888)                40.6 / 36.8  33.8 / 38.6
constexpr long long kSmallTiles = 444, kNarrowTiles = 740;
constexpr int kNarrow = 256;  // columns; up to here the two are even between the limits

struct Variant {
    int tx, ty, nthr, own;
    size_t smem;
    // order2 stage0, order2 stage1, order1, MUSCL-Hancock order2, MUSCL-Hancock order1
    void (*k[5])(Stage64Args);
};

template <int TX, int TY, int MINB, int NTHR = TX * TY, int OWN = 0>
Variant make_variant() {
    Variant v;
    v.tx = TX;
    v.ty = TY;
    v.nthr = NTHR;
    v.own = OWN;
    v.smem = Tile<TX, TY, NTHR>::smem(OWN == 2);
    v.k[0] = stage64_kernel<TX, TY, NTHR, MINB, 2, true, false, false, OWN>;
    v.k[1] = stage64_kernel<TX, TY, NTHR, MINB, 2, false, true, false, OWN>;
    v.k[2] = stage64_kernel<TX, TY, NTHR, MINB, 1, true, true, false, OWN>;
    v.k[3] = stage64_kernel<TX, TY, NTHR, MINB, 2, true, true, true, OWN>;
    v.k[4] = stage64_kernel<TX, TY, NTHR, MINB, 1, true, true, true, OWN>;
    return v;
}

// The variant of a grid of npx x npy (owned) cells; every one gives the same
// values.
const Variant &variant(int npx, int npy) {
    static const bool fixed = std::getenv("TSU_TILE64") != nullptr;
    static const Variant v = [] {
        const char *e = std::getenv("TSU_TILE64");
        if (e && !std::strcmp(e, "32x8")) return make_variant<32, 8, 2, 320, 2>();  // the default, on every grid
        if (e && !std::strcmp(e, "16x16")) return make_variant<16, 16, 2>();
        if (e && !std::strcmp(e, "16x4")) return make_variant<16, 4, 3, 192, 2>();
        if (e && !std::strcmp(e, "32x8t256")) return make_variant<32, 8, 2, 256>();
        if (e && !std::strcmp(e, "32x8t320reg")) return make_variant<32, 8, 2, 320, 0>();
        if (e && !std::strcmp(e, "32x8t320late")) return make_variant<32, 8, 2, 320, 1>();
        // default: 32 x 8 tile, 320 threads, 2 CTAs per SM (shared memory
        // allows 2; 20 warps per SM at 96 registers), the second stage's U^n
        // and extrema staged by TMA (OWN = 2, 111 KB of shared memory per CTA).
        return make_variant<32, 8, 2, 320, 2>();
    }();
    // Small grids: 16 x 4 tiles of 192 threads.  Every phase of a tile is then
    // one round of its six warps (the 32 x 8 tile needs two of its ten).
    static const Variant small = make_variant<16, 4, 3, 192, 2>();
    const long long tiles = (long long)((npx + 15) / 16) * ((npy + 3) / 4);
    return (!fixed && tiles <= (npx <= kNarrow ? kNarrowTiles : kSmallTiles)) ? small : v;
}

}  // namespace

cudaError_t stage64_prepare(int npx, int npy) {
    const Variant &v = variant(npx, npy);
    for (int i = 0; i < 5; i++) {
        cudaError_t e = cudaFuncSetAttribute(v.k[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

bool stage64_tma_maps(const double *bufA, const double *bufB, const unsigned char *mask, const double *const ext[3],
                      long long pitch, long long plane, int npx, int npy, CUtensorMap *tmA, CUtensorMap *tmB,
                      CUtensorMap *tmM, CUtensorMap *tmO, CUtensorMap tmE[3], int rows) {
    EncodeTiledFn f = tensor_map_encoder();
    const Variant &v = variant(npx, rows);
    if (!f || npx < v.tx + 4 || npy < v.ty + 4) return false;
    if (reinterpret_cast<uintptr_t>(bufA) % 16 || reinterpret_cast<uintptr_t>(bufB) % 16 ||
        reinterpret_cast<uintptr_t>(mask) % 16 || pitch % 16)
        return false;
    for (int k = 0; k < 3; k++)
        if (reinterpret_cast<uintptr_t>(ext[k]) % 16) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)npx, (cuuint64_t)npy, 5};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * sizeof(double), (cuuint64_t)plane * sizeof(double)};
    const cuuint32_t box[3] = {(cuuint32_t)(v.tx + 4), (cuuint32_t)(v.ty + 4), 5};
    const cuuint32_t es[3] = {1, 1, 1};
    const double *bufs[2] = {bufA, bufB};
    CUtensorMap *maps[2] = {tmA, tmB};
    for (int k = 0; k < 2; k++)
        if (f(maps[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(bufs[k]), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    const cuuint64_t mdims[2] = {(cuuint64_t)npx, (cuuint64_t)npy};
    const cuuint64_t mstrides[1] = {(cuuint64_t)pitch};
    const cuuint32_t mbox[2] = {(cuuint32_t)(v.tx + 32), (cuuint32_t)(v.ty + 4)};  // Tile::MLX, LY
    if (f(tmM, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<unsigned char *>(mask), mdims, mstrides, mbox, es,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    const cuuint32_t obox[3] = {(cuuint32_t)v.tx, (cuuint32_t)v.ty, 5};
    if (f(tmO, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(bufA), dims, strides, obox, es,
          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    for (int k = 0; k < 3; k++)
        if (f(&tmE[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double *>(ext[k]), dims, strides, obox, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    return true;
}

dim3 stage64_grid(int npx, int npy) {
    const Variant &v = variant(npx, npy);
    return dim3((npx + v.tx - 1) / v.tx, (npy + v.ty - 1) / v.ty);
}

cudaError_t stage64_launch(int order, int stage, const Stage64Args &a, cudaStream_t st) {
    const Variant &v = variant(a.phys.npx, a.phys.npy);
    dim3 g = stage64_grid(a.phys.npx, a.phys.npy);
    int which = (order == 2) ? (stage == 0 ? 0 : 1) : 2;
    if (a.phys.rk == 0) which = (order == 2) ? 3 : 4;  // MUSCL-Hancock: one stage
    return launch_after(v.k[which], g, dim3(v.nthr), v.smem, st, a);
}

cudaError_t initial_dt_launch(const double *V, long long pitch, long long plane, const Phys64 &P, double *partials,
                              unsigned *ticket, double *scal, cudaStream_t st) {
    dim3 b(32, 8), g((P.npx + 31) / 32, (P.npy + 7) / 8);
    dt_partials_kernel<<<g, b, 0, st>>>(V, pitch, plane, P, partials, ticket, scal);
    return cudaGetLastError();
}

cudaError_t fill_launch(double *p, long long n, double v, cudaStream_t st) {
    fill_kernel<<<1184, 256, 0, st>>>(p, n, v);
    return cudaGetLastError();
}

cudaError_t consts_launch(const SimParams &p, TsuConsts *k, cudaStream_t st) {
    consts_kernel<<<1, 1, 0, st>>>(p, k);
    return cudaGetLastError();
}

size_t partials_needed(int npx, int npy) {
    // enough for every tile shape and for the 32x8 initial-dt grid
    size_t a = (size_t)((npx + 15) / 16) * ((npy + 3) / 4);
    size_t b = (size_t)((npx + 31) / 32) * ((npy + 7) / 8);
    return a > b ? a : b;
}

}  // namespace tsu
