// gk_stage3d.cuh -- the 3D RK stage in two kernels (included by
// gk_kernels.cuh inside the mode namespace).
//
// k_zflux: the z-face fluxes of a state (or their differences) into F3.  The reference forms the
// z-face states with ReconstructYZPLM, whose slope is along y
// (recon_piecewise_linear.cpp:29-50): the left state of face (k-1|k) is the
// upper y state of cell (k-1, j), the right state the lower y state of cell
// (k, j).  A thread owns a column (i, j) and marches up a segment of faces,
// converting each plane's three rows to primitives (ConsToPrim,
// adiabatic.cpp:18-61) and sloping them once for the two faces the cell
// touches.
//
// k_stage3d: one z-plane of the stage, as the fused 2D stage does it --
// a CTA owns NT-4 columns plus a 2-cell halo, marches up a segment of rows,
// exchanges x neighbours through shared memory and solves each x and y face
// once -- with all five variables, and adds the z-flux divergence from F3.
// Face states, Riemann solver, flux divergence, RK combine and floors are the
// generic path's expressions (k_c2p, k_flux, k_update), so both paths give
// the same bits.
#pragma once

struct W5 {
    double v[5];  // primitive slots: rho, vx, vy, p, vz
};

__device__ __forceinline__ W5 c2p_at(const double* __restrict__ u, const Geom& g, const Phys& ph,
                                     long long c) {
    W5 w;
    cons_to_prim5(u[gk::S_DEN * g.vstride + c], u[gk::S_MTX * g.vstride + c],
                  u[gk::S_MTY * g.vstride + c], u[gk::S_MTZ * g.vstride + c],
                  u[gk::S_ENG * g.vstride + c], ph, w.v);
    return w;
}

// Raw conserved values of one cell (slot order), loaded ahead of their use
// so that the loads of the next row are in flight while this row computes.
struct Q5 {
    double q[5];
};
__device__ __forceinline__ Q5 load5(const double* __restrict__ u, const Geom& g, long long c) {
    Q5 r;
#pragma unroll
    for (int v = 0; v < 5; ++v) r.q[v] = __ldg(u + v * g.vstride + c);
    return r;
}
// `bad`: set where the density is out of parity mode's range (c2p_q redoes it)
__device__ __forceinline__ W5 c2p_q(const Q5& a, const Phys& ph, bool& bad) {
    W5 w;
    cons_to_prim5(a.q[gk::S_DEN], a.q[gk::S_MTX], a.q[gk::S_MTY], a.q[gk::S_MTZ], a.q[gk::S_ENG],
                  rcp_ranged(GK_FLOOR(a.q[gk::S_DEN], ph.dmin), bad), ph, w.v);
    return w;
}
__device__ __forceinline__ W5 c2p_q(const Q5& a, const Phys& ph) {
    W5 w;
    cons_to_prim5(a.q[gk::S_DEN], a.q[gk::S_MTX], a.q[gk::S_MTY], a.q[gk::S_MTZ], a.q[gk::S_ENG], ph,
                  w.v);
    return w;
}

// Riemann problem of a y face (vy | vz, vx), and of an x face (vx | vy, vz)
// and a y face together (see hllc_xy), hllc.cpp:25-27; the fluxes land in slot
// order (DEN, MTX, MTY, ENG, MTZ).
__device__ __forceinline__ void slots_y(const Flux5& f, double (&F)[5]) {
    F[gk::S_DEN] = f.d;
    F[gk::S_MTY] = f.n;
    F[gk::S_MTZ] = f.t1;
    F[gk::S_MTX] = f.t2;
    F[gk::S_ENG] = f.e;
}
__device__ __forceinline__ void hllc5_y(const double (&l)[5], const double (&r)[5], const Phys& ph,
                                        double (&F)[5]) {
    Flux5 f;
    hllc<true>(l[gk::P_RHO], l[gk::P_VY], l[gk::P_VZ], l[gk::P_VX], l[gk::P_PRE], r[gk::P_RHO],
                     r[gk::P_VY], r[gk::P_VZ], r[gk::P_VX], r[gk::P_PRE], ph, f);
    slots_y(f, F);
}
__device__ __forceinline__ void hllc5_xy(const double (&xl)[5], const double (&xr)[5],
                                         double (&Fx)[5], const double (&yl)[5],
                                         const double (&yr)[5], double (&Fy)[5], const Phys& ph) {
    bool badx = !ph.ranged, bady = !ph.ranged;
    HllcAux ax, ay;
    Flux5 fx, fy;
#define GK_XARGS xl[gk::P_RHO], xl[gk::P_VX], xl[gk::P_VY], xl[gk::P_VZ], xl[gk::P_PRE], \
                 xr[gk::P_RHO], xr[gk::P_VX], xr[gk::P_VY], xr[gk::P_VZ], xr[gk::P_PRE], ph, fx, badx, ax
#define GK_YARGS yl[gk::P_RHO], yl[gk::P_VY], yl[gk::P_VZ], yl[gk::P_VX], yl[gk::P_PRE], \
                 yr[gk::P_RHO], yr[gk::P_VY], yr[gk::P_VZ], yr[gk::P_VX], yr[gk::P_PRE], ph, fy, bady, ay
    hllc_ranged<true>(GK_XARGS);
    hllc_ranged<true>(GK_YARGS);
#if !GK_FASTMATH
    if (badx || bady || ax.zero || ay.zero) {
        hllc_redo<true>(GK_XARGS);
        hllc_redo<true>(GK_YARGS);
    }
#endif
#undef GK_XARGS
#undef GK_YARGS
    Fx[gk::S_DEN] = fx.d;
    Fx[gk::S_MTX] = fx.n;
    Fx[gk::S_MTY] = fx.t1;
    Fx[gk::S_MTZ] = fx.t2;
    Fx[gk::S_ENG] = fx.e;
    slots_y(fy, Fy);
}

// ------------------------------------------------------------ z faces
// Flux::CalFlux's z sweep (cal_flux.cpp:140-156; first order 72-87): PLM states and HLLC at
// every z face.  A CTA of 128 threads owns a tile of 32 columns x 4 rows of z faces and
// marches up a segment of zseg faces; a thread owns column (i, j) of the
// tile.  Per plane the CTA converts the tile's 6 rows (the 4 rows and one
// halo row below and above) once, 1.5 cells per face instead of the 3 a
// thread converting its own rows j-1, j, j+1 would, into a double-buffered
// shared array; the raw values of the next plane are in flight while a face
// is solved.  The y-slope of cell (k, j) gives both its lower state (the
// right state of face k-1|k) and its upper state (the left state of face
// k|k+1).  The expressions are k_flux's, so the fluxes are the same bits.
// Fast mode writes each cell's difference of its two z fluxes, the term the
// update takes (a segment's first face is solved by the segment below too): the
// x-y stage reads 5 values per cell instead of 10 and holds 10 registers less
// (256^3: 2.07 -> 2.02 ms per step).  Parity mode, whose x-y stage loads them
// late and spills differently, is faster with the fluxes (192^3: 1.74 ms, 1.82
// with differences).
constexpr int kZX = 32, kZY = 4, kZRows = kZY + 2, kZCells = kZX * kZRows;

constexpr bool kZDiff = GK_FASTMATH;
template <bool PLM>
__global__ void __launch_bounds__(128)
    k_zflux(const double* __restrict__ u, double* __restrict__ F3, Geom g, Phys ph,
            const DevTime* __restrict__ tm, int zseg) {
    if (!tm->active) return;
    __shared__ double sW[2][kZRows][5][kZX];
    const int t = threadIdx.x, tx = t & (kZX - 1), ty = t / kZX;
    const int i = g.ib + blockIdx.x * kZX + tx;
    const int j = g.jb + blockIdx.y * kZY + ty;
    const bool mine = i < g.ie && j < g.je;
    const int k0 = g.kb + blockIdx.z * zseg;  // the first face (k0-1 | k0), and the last
    const int k1 = kZDiff ? min(k0 + zseg, g.ke) : min(k0 + zseg, g.ke + 1) - 1;
    // the cells this thread loads: m = t and m = t + 128 (< 192) of the tile's
    // 6 x 32 cells, rows j0-1 .. j0+4 (clamped into the array: rows and
    // columns past the grid feed no face of this tile)
    const int j0 = g.jb + blockIdx.y * kZY;
    auto cell_of = [&](int m) {
        const int row = min(j0 - 1 + m / kZX, g.leny - 1);
        const int col = min(g.ib + blockIdx.x * kZX + (m % kZX), g.lenx - 1);
        return sidx(g, g.kb, row, col) - sidx(g, g.kb, 0, 0);  // offset within a plane
    };
    const long long off0 = cell_of(t);
    const bool two = t + 128 < kZCells;
    const long long off1 = two ? cell_of(t + 128) : off0;
    auto load = [&](int k, Q5& a, Q5& b) {
        const long long base = sidx(g, k, 0, 0);
        a = load5(u, g, base + off0);
        if (two) b = load5(u, g, base + off1);
    };
    auto put = [&](int buf, int m, const Q5& q) {
        const W5 w = c2p_q(q, ph);
#pragma unroll
        for (int v = 0; v < 5; ++v) sW[buf][m / kZX][v][m % kZX] = w.v[v];
    };
    // states of cell (k, j) from the tile's rows ty, ty+1, ty+2 (= j-1, j, j+1)
    auto states = [&](int buf, double (&lo)[5], double (&up)[5]) {
        double a[5], b[5], c[5], h[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            a[v] = sW[buf][ty][v][tx];
            b[v] = sW[buf][ty + 1][v][tx];
            c[v] = sW[buf][ty + 2][v][tx];
        }
        if (PLM) half_slopes5(a, b, c, h);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            lo[v] = PLM ? b[v] - h[v] : b[v];
            up[v] = PLM ? b[v] + h[v] : b[v];
        }
    };
    Q5 qa, qb;
    double wl[5], wr[5], nu[5], below[5];
    load(k0 - 1, qa, qb);
    put(0, t, qa);
    if (two) put(0, t + 128, qb);
    load(k0, qa, qb);
    __syncthreads();
    states(0, wr, wl);  // the upper state of plane k0-1 is the first face's left state
    int buf = 1;
    for (int k = k0; k <= k1; ++k) {
        put(buf, t, qa);
        if (two) put(buf, t + 128, qb);
        if (k < k1) load(k + 1, qa, qb);
        __syncthreads();  // plane k in sW[buf]; sW[buf ^ 1] is free for plane k+1
        states(buf, wr, nu);
        if (mine) {
            // z face (k-1 | k): (vz | vx, vy)
            Flux5 f;
            hllc<true>(wl[gk::P_RHO], wl[gk::P_VZ], wl[gk::P_VX], wl[gk::P_VY],
                             wl[gk::P_PRE], wr[gk::P_RHO], wr[gk::P_VZ], wr[gk::P_VX],
                             wr[gk::P_VY], wr[gk::P_PRE], ph, f);
            double fz[5];
            fz[gk::S_DEN] = f.d;
            fz[gk::S_MTZ] = f.n;
            fz[gk::S_MTX] = f.t1;
            fz[gk::S_MTY] = f.t2;
            fz[gk::S_ENG] = f.e;
            if (!kZDiff || k > k0) {
                const long long c = fidx(g, kZDiff ? k - 1 : k, j, i);
#pragma unroll
                for (int v = 0; v < 5; ++v) F3[v * g.fvstride + c] = kZDiff ? fz[v] - below[v] : fz[v];
            }
#pragma unroll
            for (int v = 0; v < 5; ++v) below[v] = fz[v];
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) wl[v] = nu[v];
        buf ^= 1;
    }
}

// An 8-byte copy from global to the thread's own shared word, in flight until
// copies_wait (no registers, no barrier).  The x-y stage's row inputs held 15-20
// doubles in registers in fast mode (256^3: 2.01 -> 1.99 ms per step without) and
// were loaded at their use in parity mode.
__device__ __forceinline__ void copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------ x-y plane stage
// THREE = false: out = c1*uc - c2*dF (stage 1); true: out = c1*u0 + c2*uc -
// c3*dF.  out never aliases uc (neighbours of uc are read while out is
// written); u0 may alias out (read pointwise, before the write).  LAST: the
// step's last stage also reduces the CFL speed of the new state (CalCmax,
// adiabatic.cpp:115-160, on the values it writes) and its last CTA runs the
// step epilogue, as k_cfl would after it.
// Resident threads per SM: 384, at up to 168 registers each (parity mode with
// 64-96 bytes of spills in 3D, 44-84 in 2D).  Parity mode at 192^3: 1.74 ms per step, 1.72 at 256
// threads without spills, which loses 10-30 % on small grids (64^3: 158 us
// against 207); fast mode at 512 threads (128 registers, no spills) is no faster
// at 256^3 (2.175 -> 2.162 ms) and slower on small grids (31x190x55 82 -> 88 us).
constexpr int kStage3dThreadsPerSM = 384;
// ZF = false: a 2D run with all five variables (one plane, no z fluxes): the
// update is k_update's 2D expression.  A 2D run off the four-variable path
// (v_z, z gravity, point masses, an immersed body) took five launches per
// stage through primitive and flux arrays; this is one.
// LAST = 2: the second half kick of constant gravity and one point mass too.
template <int NT, bool THREE, bool PLM, int LAST, bool ZF>
__global__ void __launch_bounds__(NT, kStage3dThreadsPerSM / NT)
    k_stage3d(const double* __restrict__ uc, const double* u0, double* out,
              const double* __restrict__ F3, Geom g, Phys ph, double c1, double c2, double c3,
              DevTime* tm, int rows, int has_z) {
    if (!tm->active) return;
    unsigned long long cbest = 0ull;  // CFL speed of this thread's cells (bit pattern)
    __shared__ double sP[5][NT];
    __shared__ double sXL[5][NT];
    __shared__ double sF[5][NT];
    // rows of sIn: z-flux difference or lower z flux, raw state, base state, upper z flux
    constexpr int kB0 = ZF ? 5 : 0, kIn = kB0 + (THREE ? 10 : 5) + (ZF && !kZDiff ? 5 : 0);
    __shared__ double sIn[kIn][NT];
    const double dt = tm->dt;
    const double dtdx = dt * g.dxRec, dtdy = dt * g.dyRec, dtdz = dt * g.dzRec;
    const int t = threadIdx.x;
    const int tl = t > 0 ? t - 1 : 0;
    const int tr = t < NT - 1 ? t + 1 : t;
    const int xi = g.ib - 2 + blockIdx.x * (NT - 4) + t;
    const int xl = xi < g.lenx ? xi : g.lenx - 1;  // clamped load column
    const bool do_cell = t >= 2 && t <= NT - 3 && xi < g.ie;
    const int k = g.kb + blockIdx.z;
    const int y0 = g.jb + blockIdx.y * rows;
    const int y1 = min(y0 + rows, g.je);
    auto at = [&](int j) { return sidx(g, k, j, xl); };

    // primitives of rows y0-2, y0-1, y0 and y0+1
    const W5 Pm2 = c2p_at(uc, g, ph, at(y0 - 2));
    W5 Pm1 = c2p_at(uc, g, ph, at(y0 - 1));
    W5 P0 = c2p_at(uc, g, ph, at(y0));
    double wlNext[5], fyPrev[5];
    // lower state of y face y0 (upper y state of cell y0-1), then that face
    {
        const W5 P1 = c2p_at(uc, g, ph, at(y0 + 1));
        double wr[5], h[5], h0[5];
        if (PLM) {
            half_slopes5(Pm2.v, Pm1.v, P0.v, h);
            half_slopes5(Pm1.v, P0.v, P1.v, h0);
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            wlNext[v] = PLM ? Pm1.v[v] + h[v] : Pm1.v[v];
            wr[v] = PLM ? P0.v[v] - h0[v] : P0.v[v];
        }
        hllc5_y(wlNext, wr, ph, fyPrev);
#pragma unroll
        for (int v = 0; v < 5; ++v) wlNext[v] = PLM ? P0.v[v] + h0[v] : P0.v[v];
        Pm1 = P0;
        P0 = P1;
    }
    // row f: the x faces of cell row f-1 and the y face f above it; update row f-1.
    // The raw row f+2 is loaded one row ahead of its conversion.
    Q5 Qn = load5(uc, g, at(y0 + 2));
    for (int f = y0 + 1; f <= y1; ++f) {
        const Q5 Q1 = Qn;
        if (f + 2 <= y1 + 1) Qn = load5(uc, g, at(f + 2));
        // what the update of cell row f-1 takes beside the fluxes: its z fluxes
        // (or their difference), base state and raw state, copied to this
        // thread's own shared words while the row's Riemann problems are solved
        if (do_cell) {
            const long long fc = ZF ? fidx(g, k, f - 1, xi) : 0;
            const long long c = at(f - 1);
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                if (ZF) copy8(&sIn[v][t], F3 + v * g.fvstride + fc);
                if (ZF && !kZDiff) copy8(&sIn[kIn - 5 + v][t], F3 + v * g.fvstride + fc + g.fkstride);
                copy8(&sIn[kB0 + v][t], uc + v * g.vstride + c);
                if (THREE) copy8(&sIn[kB0 + 5 + v][t], u0 + v * g.vstride + c);
            }
        }
        bool bad;  // parity mode: a quotient of this phase is out of range
        SlopeRange rg;
        clear(rg);
        W5 P1 = c2p_q(Q1, ph, bad);
#pragma unroll
        for (int v = 0; v < 5; ++v) sP[v][t] = Pm1.v[v];
        __syncthreads();
        double xr[5], wr[5], wlNew[5], hx[5], hy[5];
        if (PLM) {
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                hx[v] = vanleer_half(Pm1.v[v] - sP[v][tl], sP[v][tr] - Pm1.v[v], rg);
                hy[v] = vanleer_half(P0.v[v] - Pm1.v[v], P1.v[v] - P0.v[v], rg);
            }
        }
#if !GK_FASTMATH
        if (bad || (PLM && out_of_range(rg))) {
            P1 = c2p_q(Q1, ph);
            if (PLM) {
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    hx[v] = vanleer_half_any(Pm1.v[v] - sP[v][tl], sP[v][tr] - Pm1.v[v]);
                    hy[v] = vanleer_half_any(P0.v[v] - Pm1.v[v], P1.v[v] - P0.v[v]);
                }
            }
        }
#endif
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            if (PLM) {
                sXL[v][t] = Pm1.v[v] + hx[v];
                xr[v] = Pm1.v[v] - hx[v];
                wr[v] = P0.v[v] - hy[v];
                wlNew[v] = P0.v[v] + hy[v];
            } else {
                sXL[v][t] = Pm1.v[v];
                xr[v] = Pm1.v[v];
                wr[v] = P0.v[v];
                wlNew[v] = P0.v[v];
            }
        }
        __syncthreads();
        double xlst[5], fx[5], fy[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) xlst[v] = sXL[v][tl];
        hllc5_xy(xlst, xr, fx, wlNext, wr, fy, ph);
#pragma unroll
        for (int v = 0; v < 5; ++v) sF[v][t] = fx[v];
        __syncthreads();
        if (do_cell) {
            // update_cons.cpp (3D): (Fx(i+1)-Fx(i))*dtdx + (Fy(j+1)-Fy(j))*dtdy + (Fz(k+1)-Fz(k))*dtdz
            copies_wait();
            const long long c = at(f - 1);
            double r[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
#if GK_FASTMATH
                double dF = (sF[v][tr] - fx[v]) * dtdx + (fy[v] - fyPrev[v]) * dtdy;
                if (ZF) dF += (kZDiff ? sIn[v][t] : sIn[kIn - 5 + v][t] - sIn[v][t]) * dtdz;
                r[v] = stage_value<THREE>(c1, c2, c3, THREE ? sIn[kB0 + 5 + v][t] : 0.0, sIn[kB0 + v][t], dF);
#else
                double dF = (sF[v][tr] - fx[v]) * dtdx;
                if (ZF) dF = dF + (fy[v] - fyPrev[v]) * dtdy +
                             (kZDiff ? sIn[v][t] : sIn[kIn - 5 + v][t] - sIn[v][t]) * dtdz;
                else dF = dF + (fy[v] - fyPrev[v]) * dtdy;
                if (THREE) r[v] = c1 * sIn[kB0 + 5 + v][t] + c2 * sIn[kB0 + v][t] - c3 * dF;
                else r[v] = c1 * sIn[kB0 + v][t] - c2 * dF;
#endif
            }
            constexpr bool SPEED = ZF && LAST == 1;
            const double speed = floors5_speed<SPEED>(r, ph, tm);
            if (LAST) {
                if (LAST == 2) kick_cell<false>(r, g, ph, dt, tm->t, 1, xi, f - 1, k);
                const double local = SPEED ? speed
                                           : cell_cmax(r[gk::S_DEN], r[gk::S_MTX], r[gk::S_MTY],
                                                       r[gk::S_MTZ], r[gk::S_ENG], ph, ZF || has_z);
                const unsigned long long b = (unsigned long long)__double_as_longlong(local);
                cbest = b > cbest ? b : cbest;
            }
#pragma unroll
            for (int v = 0; v < 5; ++v) out[v * g.vstride + c] = r[v];
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            fyPrev[v] = fy[v];
            wlNext[v] = wlNew[v];
        }
        Pm1 = P0;
        P0 = P1;
    }
    if (LAST) last_stage_end<NT>(cbest, tm, g, ph, gridDim.x * gridDim.y * gridDim.z);
}

// ------------------------------------------------------------ long 1D rows
// One RK stage of a 1D run in one launch: the x part of k_stage3d on one row,
// each CTA of 128 threads updating 124 cells, with the x sides' ghost fill in
// the CTAs that hold ghosts (they also write them back: a frame's ghost strips
// come from there).  KIND 0: out = c1*uc - c2*dF; 1: out = c1*u0 + c2*uc -
// c3*dF; 2: as 1, the step's last stage (CFL reduction and epilogue); 3: with
// the second half kick too.  The expressions are the per-phase kernels'
// (k_c2p, k_flux, k_update, k_kick, k_cfl), so the bits are the same; those
// took 11 launches per RK2 step and converted every ghost row of the array
// (262143 cells, parity: 90 us per step; FP64 alone needs 9).
// CTAS: resident CTAs per SM.  A row with tiles for more than three per SM hides
// its latency better with more, at fewer registers and without spills (5 in fast
// mode, 4 in parity mode, which needs 128): 262143 cells, us per step, fast 18.5 ->
// 17.2, parity 25.7 -> 24.4; 2^20 cells fast 53.1 -> 50.2.  Shorter rows keep three
// (1100 cells, parity: 10.2, at four 10.35).
constexpr int kRowThreads = 128, kRowCtas = 3, kRowCtasLong = GK_FASTMATH ? 5 : 4;
template <int KIND, bool PLM, int CTAS>
__global__ void __launch_bounds__(kRowThreads, CTAS)
    k_row_stage(double* uc, const double* u0, double* out, Geom g, Phys ph, double c1, double c2,
                double c3, DevTime* tm, int has_z, int tiles) {
    if (!tm->active) return;
    constexpr int NT = kRowThreads;
    constexpr bool THREE = KIND >= 1, LAST = KIND >= 2;
    __shared__ double sP[5][NT];
    __shared__ double sXL[5][NT];
    __shared__ double sF[5][NT];
    const int t = threadIdx.x;
    const int tl = t > 0 ? t - 1 : 0;
    const int tr = t < NT - 1 ? t + 1 : t;
    const double dtdx = tm->dt * g.dxRec;
    // raw state and base state of this thread's cell of a tile, ghosts filled
    auto load = [&](int tile, Q5& q, double (&b0)[5]) {
        const int xi = g.ib - 2 + tile * (NT - 4) + t;
        if (xi < g.ib || (xi >= g.ie && xi < g.lenx))
            bc_fill_one(uc, g, ph, 0, xi >= g.ie, xi < g.ib ? xi : xi - g.ie);
        const long long c = sidx(g, g.kb, g.jb, xi < g.lenx ? xi : g.lenx - 1);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            q.q[v] = uc[v * g.vstride + c];
            if (THREE) b0[v] = u0[v * g.vstride + c];
        }
    };
    Q5 qn;
    double bn[5];
    load(blockIdx.x, qn, bn);
    unsigned long long cbest = 0ull;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int xi = g.ib - 2 + tile * (NT - 4) + t;
        const bool do_cell = t >= 2 && t <= NT - 3 && xi < g.ie;
        const Q5 q = qn;
        double b0[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) b0[v] = bn[v];
        if (tile + (int)gridDim.x < tiles) load(tile + gridDim.x, qn, bn);  // arrives meanwhile
        const W5 P = c2p_q(q, ph);
#pragma unroll
        for (int v = 0; v < 5; ++v) sP[v][t] = P.v[v];
        __syncthreads();
        double xr[5];
        if (PLM) {
            double a[5], d[5], h[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                a[v] = sP[v][tl];
                d[v] = sP[v][tr];
            }
            half_slopes5(a, P.v, d, h);
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                sXL[v][t] = P.v[v] + h[v];
                xr[v] = P.v[v] - h[v];
            }
        } else {
#pragma unroll
            for (int v = 0; v < 5; ++v) sXL[v][t] = xr[v] = P.v[v];
        }
        __syncthreads();
        Flux5 f;
        hllc<true>(sXL[gk::P_RHO][tl], sXL[gk::P_VX][tl], sXL[gk::P_VY][tl],
                         sXL[gk::P_VZ][tl], sXL[gk::P_PRE][tl], xr[gk::P_RHO], xr[gk::P_VX],
                         xr[gk::P_VY], xr[gk::P_VZ], xr[gk::P_PRE], ph, f);
        double fx[5];
        fx[gk::S_DEN] = f.d;
        fx[gk::S_MTX] = f.n;
        fx[gk::S_MTY] = f.t1;
        fx[gk::S_MTZ] = f.t2;
        fx[gk::S_ENG] = f.e;
#pragma unroll
        for (int v = 0; v < 5; ++v) sF[v][t] = fx[v];
        __syncthreads();
        if (do_cell) {
            double r[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                const double dF = (sF[v][tr] - fx[v]) * dtdx;
                if (THREE) r[v] = c1 * b0[v] + c2 * q.q[v] - c3 * dF;
                else r[v] = c1 * q.q[v] - c2 * dF;
            }
            floors5(r, ph, tm);
            if (LAST) {
                if (KIND == 3) kick_cell<false>(r, g, ph, tm->dt, tm->t, 1, xi, g.jb, g.kb);
                const unsigned long long b = (unsigned long long)__double_as_longlong(
                    cell_cmax(r[gk::S_DEN], r[gk::S_MTX], r[gk::S_MTY], r[gk::S_MTZ], r[gk::S_ENG], ph,
                              has_z));
                cbest = b > cbest ? b : cbest;
            }
            const long long c = sidx(g, g.kb, g.jb, xi);
#pragma unroll
            for (int v = 0; v < 5; ++v) out[v * g.vstride + c] = r[v];
        }
    }
    if (LAST) last_stage_end<NT>(cbest, tm, g, ph, gridDim.x);
}
