// lbf_stream_kernel.cuh -- body of the fused step kernel (see lbf_stream.cuh).
//
// Per z plane q a CTA runs two barrier phases:
//   phase 1  the in-plane partials of phi(q+3) and theta(q+2) on the theta
//            region, and the moments prologue + collision of plane q on the
//            collision region (populations to shared memory).  The two sets
//            of work are independent, so one barrier covers both, and the
//            halo-ring collisions are placed on the warps with no theta work.
//            Before the barrier each thread issues the loads of its interior
//            node's fields of plane q+1.
//   phase 2  an asynchronous copy (cp.async) of phi(q+4) into its ring
//            slot; the theta partials of plane q+2; then every output node
//            pulls the populations of plane q and plane q-1 is written.  The
//            copy completes behind this phase.
#pragma once
#include "lbf_chain.cuh"
#include "lbf_node.cuh"
#include "lbf_single_kernel.cuh"

namespace lbf {

// The moments (and u_old) of a collision node go from global memory straight
// into registers: the tile-interior node's one plane ahead (NodeRaw, below),
// the ring nodes' at the point of use.  A cp.async prefetch of them into a
// shared staging area, one plane ahead, lost more than it hid: its
// shared-memory writes were bank-conflicted (13.6 M of the 19.8 M conflicts of a
// 256^3 FP32 launch) and the extra 52 B/node of shared traffic competed with the
// population exchange; without it the FP32 Laplace step ran 14.1 against 12.0
// GLUPS.

// ring slots of the separable phase-field stencils (see step_body)
constexpr int SXY_SLOTS = 5, GXY_SLOTS = 3, TH_SLOTS = 2, GT_SLOTS = 3, H_SLOTS = 3;

// asynchronous global -> shared copies of 4 or 8 bytes
template <int BYTES> __device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    if constexpr (BYTES == 4) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
    }
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <typename S, typename R, int TYV> constexpr size_t stream_smem_bytes() {
    constexpr int R1N = Tile<TYV>::R1N, R2N = Tile<TYV>::R2N, R3N = Tile<TYV>::R3N;
    size_t b = sizeof(R) * size_t(24) * R1N;  // populations: 8 (cx, cy) groups x 3 cz (the centre stays in registers)
    b += sizeof(R) * (size_t(PHI_SLOTS) * R3N + size_t(SXY_SLOTS) * R2N + size_t(GXY_SLOTS) * 2 * R2N +
                          size_t(TH_SLOTS) * 3 * R2N + size_t(GT_SLOTS) * 3 * R1N + size_t(H_SLOTS) * 3 * R1N);
    return b;
}

// One piece of a time step: tile (bx, by) of the box, planes z0 <= z < z1.
// REP: REPULSIVE_FLUX force in the moments prologue; OBS: 1 obstacles (isfluid
// tests, the moment-space bounce-back) and the phi mass correction, 2 the
// correction alone, 0 neither; 3 the code of 1 for a box without obstacles (a
// batch's), which takes the HIGHORDER rows in the form that such a box steps
// with alone.  Separate compilations, so the kernels without
// them carry no code for them: the obstacle code alone, never executed, costs a
// box without obstacles 5.6 %, and the correction in that compilation a quarter
// of the step (150 x 128 x 136: 257 us with its sum, 214 us in a compilation of
// its own).
template <int LAT, bool HO, typename S, typename R, int TYV, bool REP, int OBS>
__device__ __forceinline__ void step_body(const StepParams<S, R>& p, const int bx, const int by, const int z0,
                                          const int z1) {
    using TL = Tile<TYV>;
    constexpr int TY = TL::TY, NT = TL::NT, NRING1 = TL::NRING1, NTH = TL::NTH, KTH = TL::KTH;
    constexpr int R1Y = TL::R1Y, R1N = TL::R1N, R2Y = TL::R2Y, R2N = TL::R2N, R3N = TL::R3N;
    using CD = Codec<S>;
    using SP = typename PhiStore<S>::type;
    using CP = Codec<SP>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // post-collision populations of plane q, by (cx, cy) group g = 3 (cy+1) + (cx+1):
    // the output nodes that read one group of a node read all three cz of it
    using R2 = typename Vec2<R>::type;
    // (the centre group (0, 0) of a node is read only by the node's own
    // output, the thread that collided it: it stays in registers)
    R2* pops2 = reinterpret_cast<R2*>(smem_raw);                  // [8][R1N] (cz = -1, cz = 0)
    R* pops1 = reinterpret_cast<R*>(pops2 + 8 * R1N);             // [8][R1N] (cz = +1)
    R* phis = pops1 + 8 * R1N;                         // [PHI_SLOTS][R3N]
    auto gslot = [](int g) { return g < 4 ? g : g - 1; };  // shared slot of group g != 4
    auto put_group = [&](int g, int node, R vm, R v0, R vp) {
        R2 v;
        v.x = vm;
        v.y = v0;
        pops2[gslot(g) * R1N + node] = v;
        pops1[gslot(g) * R1N + node] = vp;
    };
    R* sxys = phis + PHI_SLOTS * R3N;       // [SXY_SLOTS][R2N] S_x S_y phi
    R* gxys = sxys + SXY_SLOTS * R2N;       // [GXY_SLOTS][2][R2N] D_x S_y phi, S_x D_y phi
    R* ths = gxys + GXY_SLOTS * 2 * R2N;    // [TH_SLOTS][3][R2N] theta
    R* gts = ths + TH_SLOTS * 3 * R2N;      // [GT_SLOTS][3][R1N] g~
    R* hs = gts + GT_SLOTS * 3 * R1N;       // [H_SLOTS][3][R1N] theta partials

    const int t = threadIdx.x;
    const int tx = t % TX, ty = t / TX;
    const int X0 = bx * TX, Y0 = by * TY;
    // node indices inside one field fit in 32 bits (boxes hold < 2^31 nodes);
    // field bases (f * N) are 64-bit and uniform across the CTA
    const long long N = p.N;
    const int plane = (int)p.plane;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const bool dr = p.densratio != 0;
    const bool obs = (OBS & 1) && p.obstacles != 0;
    const R cssq = R(1.0 / 3.0);

    // ---- static per-thread node tables (x/y wrap does not change along z) ----
    // collision nodes: A = tile interior node t; B = ring node r for the threads
    // of the last warps (t >= NTH), r = t - NTH < NRING1
    const int nodeA = (ty + 1) * R1X + (tx + 1);
    int nodeB = -1;
    {
        const int r = t - NTH;
        if (r >= 0 && r < NRING1) {
            // one kind of ring node per warp: the inner 32 nodes of the top row,
            // of the bottom row, then the left and right columns with the corners
            if (r < TX) nodeB = r + 1;                                              // top row
            else if (r < 2 * TX) nodeB = (R1Y - 1) * R1X + (r - TX + 1);            // bottom row
            else if (r < 2 * TX + R1Y) nodeB = (r - 2 * TX) * R1X;                  // left column
            else nodeB = (r - 2 * TX - R1Y) * R1X + (R1X - 1);                      // right column
        }
    }
    // ring nodes stream into the tile along one axis only: the rows' along y
    // (cy = +1 from the top row, -1 from the bottom), the columns' along x
    // (cx = +1 from the left, -1 from the right; corners with them).  ring_col
    // is uniform across a warp (the ring warps hold 32 row nodes each, then
    // the columns).
    const bool ring_col = (t - NTH) >= 2 * TX;
    R ring_dir = R(0);
    if (nodeB >= 0) {
        const int bx = nodeB % R1X, by = nodeB / R1X;
        ring_dir = ring_col ? (bx == 0 ? R(1) : R(-1)) : (by == 0 ? R(1) : R(-1));
    }
    // wrapped: the node was reached across a periodic face in x or y
    auto r1_geom = [&](int node, int& off, bool& wrapped) -> bool {
        wrapped = false;
        if (node < 0) { off = 0; return false; }
        int hx = node % R1X, hy = node / R1X;
        bool ok = true;
        const int gx0 = X0 + hx - 1, gy0 = Y0 + hy - 1;
        int gx = wrap_coord(gx0, nx, p.pbx, ok);
        int gy = wrap_coord(gy0, ny, p.pby, ok);
        wrapped = gx != gx0 || gy != gy0;
        off = ok ? gy * nx + gx : 0;
        return ok;
    };
    int offA, offB;
    bool wrapA, wrapB;
    const bool okA = r1_geom(nodeA, offA, wrapA);
    const bool okB = r1_geom(nodeB, offB, wrapB);
    // phi mass correction of the input phi
    double mcorr = 0.0;
    bool do_mcorr = false;
    if constexpr (OBS) do_mcorr = mass_corr(p.mass, mcorr);
    const int ox = X0 + tx, oy = Y0 + ty;
    const bool out_ok = (ox < nx) && (oy < ny);
    const int out_off = oy * nx + ox;


    // theta nodes (R2): slot n = t + k NTH of the first NTH threads; phi nodes
    // (R3): t, t + NT, t + 2 NT.  Slot n maps to the first TX columns of each
    // row of the theta region, one row per warp, then to the remaining
    // R2X - TX columns of every row: a warp's loads from the rings then stay
    // in one row, 32 consecutive words, instead of straddling two rows of the
    // wider rings (a two-way bank conflict).  Storage stays row-major.
    auto r2_node = [](int n, int& hx, int& hy) {
        constexpr int MAIN = TX * Tile<TYV>::R2Y;
        if (n < MAIN) {
            hy = n / TX; hx = n % TX;
        } else {
            const int e = n - MAIN;
            hy = e / (R2X - TX); hx = TX + e % (R2X - TX);
        }
    };
    int r2_off[KTH];
    bool r2_ok[KTH];
#pragma unroll
    for (int k = 0; k < KTH; ++k) {
        r2_off[k] = 0;
        r2_ok[k] = false;
    }
    int r3_off[3] = {0, 0, 0};
    bool r3_ok[3] = {false, false, false};
#pragma unroll
    for (int k = 0; k < KTH; ++k) {
        int n = t + k * NTH;
        if (t < NTH && n < R2N) {
            int hx, hy;
            r2_node(n, hx, hy);
            bool ok = true;
            int gx = wrap_coord(X0 + hx - 2, nx, p.pbx, ok);
            int gy = wrap_coord(Y0 + hy - 2, ny, p.pby, ok);
            r2_ok[k] = ok;
            r2_off[k] = ok ? gy * nx + gx : 0;
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int n = t + k * NT;
        if (n < R3N) {
            int hx = n % R3X, hy = n / R3X;
            bool ok = true;
            int gx = wrap_coord(X0 + hx - 3, nx, p.pbx, ok);
            int gy = wrap_coord(Y0 + hy - 3, ny, p.pby, ok);
            r3_ok[k] = ok;
            r3_off[k] = ok ? gy * nx + gx : 0;
        }
    }

    auto zwrap = [&](int q, bool& ok) { return wrap_coord(q, nz, p.pbz, ok); };
    auto phi_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)PHI_SLOTS); };
    auto sxy_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)SXY_SLOTS); };
    auto gxy_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)GXY_SLOTS); };
    auto th_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)TH_SLOTS); };
    auto gt_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)GT_SLOTS); };
    auto h_slot = [&](int q) { return (int)((unsigned)(q - z0 + 3) % (unsigned)H_SLOTS); };
    // D1Q3 weights: the D3Q27 weights of the isotropic stencils factor as W(cx) W(cy) W(cz)
    const R W0 = R(2.0 / 3.0), W1 = R(1.0 / 6.0);

    // phi plane q into its ring slot (zero outside the box); asynchronous or direct
    auto load_phi_plane = [&](int q, bool async) {
        bool zok = true;
        const int wz = zwrap(q, zok);
        R* dst = phis + phi_slot(q) * R3N;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int n = t + k * NT;
            if (n < R3N) {
                const bool ok = zok && r3_ok[k];
                const int g = wz * plane + r3_off[k];
                if (async && ok) {
                    cp_async<sizeof(SP)>(dst + n, p.pin + g);
                } else {
                    dst[n] = ok ? CP::ld(p.pin, g, R(1)) : R(0);
                }
            }
        }
    };
    // Separable phase-field stencils.  The isotropic gradient, Laplacian and
    // divergence of the reference (lb_cuda_auxfields_module.f90:72-135,
    // 1136-1157) use the D3Q27 weights w = W(cx) W(cy) W(cz), W(0) = 2/3,
    // W(+-1) = 1/6, so each is a product of 1-D operators: S = W-weighted sum,
    // D = W(1) x central difference.  Per plane the theta region keeps the
    // in-plane partials S_x S_y phi, D_x S_y phi, S_x D_y phi; the z operator
    // then combines three planes of them at the same (x, y):
    //   grad phi = 3 (S_z D_x S_y, S_z S_x D_y, D_z S_x S_y) phi
    //   lap phi  = 6 (S_z S_x S_y phi - phi)
    // and likewise div theta = 3 (S_z (D_x S_y th_x + S_x D_y th_y) + D_z S_x S_y th_z)
    // from in-plane partials of theta on the collision region.  The same sums
    // as the reference, in another order.  The in-plane smoothings are kept
    // relative to the node's own value (S_x S_y f - f_c, from the differences
    // f - f_c), and z differences are taken of those and of the centre values
    // separately: a z difference of two smoothed planes of values near 1
    // would lose the digits that a small gradient needs in FP32.

    // in-plane partials of phi(q) on this thread's theta-region nodes
    auto planar_plane = [&](int q) {
        const R* f = phis + phi_slot(q) * R3N;
        R* sx = sxys + sxy_slot(q) * R2N;
        R* gg = gxys + gxy_slot(q) * (2 * R2N);
#pragma unroll
        for (int k = 0; k < KTH; ++k) {
            const int n = t + k * NTH;
            if (t >= NTH || n >= R2N) continue;
            int hx, hy;
            r2_node(n, hx, hy);
            const int m = hy * R2X + hx;
            const R* c = f + (hy + 1) * R3X + (hx + 1);
            const R fc = c[0];
            R sr[3], dr_[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const R a = c[(r - 1) * R3X - 1], b = c[(r - 1) * R3X], e = c[(r - 1) * R3X + 1];
                sr[r] = W1 * ((a - fc) + (e - fc)) + W0 * (b - fc);
                dr_[r] = e - a;
            }
            sx[m] = W1 * (sr[0] + sr[2]) + W0 * sr[1];  // S_x S_y phi - phi_c
            gg[m] = W1 * (W1 * (dr_[0] + dr_[2]) + W0 * dr_[1]);
            gg[R2N + m] = W1 * (sr[2] - sr[0]);
        }
    };
    // theta = phi(1-phi) n on the theta region and g~ = n |g| on the collision
    // region of plane q (compute_norm_interface, lb_cuda_auxfields_module.f90:72-119)
    // from the partials of planes q-1..q+1
    // Obstacles: isfluid of this thread's theta nodes in plane q (0 outside
    // the box), loaded a plane before theta_plane uses it so the load's
    // latency passes behind the pull phase; a load at the point of use
    // stalled every theta warp at once (a box with obstacles stepped 33 %
    // slower than without, with no solid node)
    auto theta_isf = [&](int q, int8_t (&s)[KTH]) {
        bool zk = true;
        const int wz = zwrap(q, zk);
#pragma unroll
        for (int k = 0; k < KTH; ++k) {
            const int n = t + k * NTH;
            s[k] = (t < NTH && n < R2N && zk && r2_ok[k]) ? p.isf[wz * plane + r2_off[k]] : int8_t(0);
        }
    };
    int8_t th_isf[KTH];
#pragma unroll
    for (int k = 0; k < KTH; ++k) th_isf[k] = 1;
    auto theta_plane = [&](int q) {
        bool zok = true;
        const int wz = zwrap(q, zok);
        const R* f0 = phis + phi_slot(q - 1) * R3N;
        const R* f1 = phis + phi_slot(q) * R3N;
        const R* f2 = phis + phi_slot(q + 1) * R3N;
        const R* s0 = sxys + sxy_slot(q - 1) * R2N;
        const R* s2 = sxys + sxy_slot(q + 1) * R2N;
        const R* g0 = gxys + gxy_slot(q - 1) * (2 * R2N);
        const R* g1 = gxys + gxy_slot(q) * (2 * R2N);
        const R* g2 = gxys + gxy_slot(q + 1) * (2 * R2N);
        R* th = ths + th_slot(q) * (3 * R2N);
        R* gt = gts + gt_slot(q) * (3 * R1N);
#pragma unroll
        for (int k = 0; k < KTH; ++k) {
            const int n = t + k * NTH;
            if (t >= NTH || n >= R2N) continue;
            int hx, hy;
            r2_node(n, hx, hy);
            const int m = hy * R2X + hx;
            bool fluid = zok && r2_ok[k];
            if (fluid && obs) fluid = (th_isf[k] == 1 || th_isf[k] == -1);
            R th0 = 0, th1 = 0, th2 = 0, gv0 = 0, gv1 = 0, gv2 = 0;
            if (fluid) {
                const R gx = R(3) * (W1 * (g0[m] + g2[m]) + W0 * g1[m]);
                const R gy = R(3) * (W1 * (g0[R2N + m] + g2[R2N + m]) + W0 * g1[R2N + m]);
                const int c3 = (hy + 1) * R3X + (hx + 1);
                const R gz = R(3) * W1 * ((s2[m] - s0[m]) + (f2[c3] - f0[c3]));
                const R mg = sqrt_a<R>(gx * gx + gy * gy + gz * gz);
                const R rden = rcp<R>(mg + R(1.0e-9));
                const R nxv = gx * rden, nyv = gy * rden, nzv = gz * rden;
                const R ph = f1[c3];
                const R pp = ph * (R(1) - ph);
                th0 = pp * nxv; th1 = pp * nyv; th2 = pp * nzv;
                gv0 = nxv * mg; gv1 = nyv * mg; gv2 = nzv * mg;
            }
            th[0 * R2N + m] = th0;
            th[1 * R2N + m] = th1;
            th[2 * R2N + m] = th2;
            if (hx >= 1 && hx <= R2X - 2 && hy >= 1 && hy <= R2Y - 2) {
                const int n1 = (hy - 1) * R1X + (hx - 1);
                gt[0 * R1N + n1] = gv0;
                gt[1 * R1N + n1] = gv1;
                gt[2 * R1N + n1] = gv2;
            }
        }
    };
    // in-plane partials of theta(q) at this thread's collision nodes:
    // D_x S_y th_x + S_x D_y th_y and S_x S_y th_z
    auto theta_partials = [&](int q) {
        const R* th = ths + th_slot(q) * (3 * R2N);
        R* h = hs + h_slot(q) * (3 * R1N);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int node = k ? nodeB : nodeA;
            if (node < 0) continue;
            const int hx = node % R1X, hy = node / R1X;
            const R* c = th + (hy + 1) * R2X + (hx + 1);
            const R zc = c[2 * R2N];
            R dx[3], sy[3], sz[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int o = (r - 1) * R2X;
                dx[r] = c[o + 1] - c[o - 1];
                sy[r] = W1 * (c[R2N + o - 1] + c[R2N + o + 1]) + W0 * c[R2N + o];
                sz[r] = W1 * ((c[2 * R2N + o - 1] - zc) + (c[2 * R2N + o + 1] - zc)) + W0 * (c[2 * R2N + o] - zc);
            }
            h[node] = W1 * (W1 * (dx[0] + dx[2]) + W0 * dx[1]) + W1 * (sy[2] - sy[0]);
            h[R1N + node] = W1 * (sz[0] + sz[2]) + W0 * sz[1];  // S_x S_y th_z - th_z,c
            h[2 * R1N + node] = zc;
        }
    };

    // stored moments, u_old and isfluid of one collision node, not yet decoded.
    // The tile-interior node's are loaded one plane ahead, at the end of the
    // collision phase of the plane before (after its collisions), so their
    // latency passes behind its barrier and the pull phase; the ring nodes
    // load theirs at the point of use.
    using LY = Layout<S>;
    struct NodeRaw {
        S m[10];      // with 16-bit storage only m[4..9] (Pi - u u)
        float v32[4];  // P, u, v, w of the 16-bit formats
        S uo[3];
        int8_t isf;
        int row;  // start of the wall links of the warp's tile row
    };
    auto fetch = [&](int gi, NodeRaw& r) {
        if constexpr (LY::split) {
#pragma unroll
            for (int f = 0; f < 4; ++f) r.v32[f] = p.pres_in[f * N + gi];
#pragma unroll
            for (int f = 4; f < 10; ++f) r.m[f] = CD::raw(p.min + LY::off(f, N), gi);
        } else {
#pragma unroll
            for (int f = 0; f < 10; ++f) r.m[f] = CD::raw(p.min + f * N, gi);
        }
        if (dr) {
#pragma unroll
            for (int f = 0; f < 3; ++f) r.uo[f] = CD::raw(p.uin + f * N, gi);
        }
        if (obs) r.isf = p.isf[gi];
    };
    NodeRaw nxt;
    auto prefetch_a = [&](int q) {
        bool zk = true;
        const int wz = zwrap(q, zk);
        if (zk && okA) fetch(wz * plane + offA, nxt);
        if (obs && q >= z0 && q < z1 && oy < ny) nxt.row = __ldg(p.link_rows + (q * ny + oy) * ((nx + TX - 1) / TX) + bx);
    };
    nxt.row = 0;

    // accumulators of the raw moments {sum g, sum g c, sum g c c} for output planes
    // q-1 (am), q (a0), q+1 (ap); A2[i] = (am[i], a0[i]), one pair, accumulated
    // with packed instructions from the population pairs (cz = -1, 0).  With
    // the packed x and y transforms of the collision: 2.9 % fewer
    // instructions, 1.8 % per step at 256^3
    using PA = typename PK<R>::T;
    PA A2[10];
    R ap[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        A2[i] = PK<R>::mk(R(0), R(0));
        ap[i] = R(0);
    }

    // ---- prologue: phi(z0-3..z0+2), theta(z0-2..z0) ----
    // partials of phi(z0-3..z0+1), theta(z0-2..z0), theta partials (z0-2, z0-1)
    // (theta reads only this thread's own partials; the partial slots are
    // reused as soon as a theta plane no longer needs them)
    for (int q = z0 - 3; q <= z0 + 1; ++q) load_phi_plane(q, false);
    __syncthreads();
    planar_plane(z0 - 3);
    planar_plane(z0 - 2);
    planar_plane(z0 - 1);
    if (obs) theta_isf(z0 - 2, th_isf);
    theta_plane(z0 - 2);
    planar_plane(z0);
    if (obs) theta_isf(z0 - 1, th_isf);
    theta_plane(z0 - 1);
    planar_plane(z0 + 1);
    __syncthreads();
    theta_partials(z0 - 2);
    theta_partials(z0 - 1);
    __syncthreads();
    if (obs) theta_isf(z0, th_isf);
    theta_plane(z0);               // into the slot of theta(z0-2)
    if (obs) theta_isf(z0 + 1, th_isf);  // for the loop's first theta plane
    load_phi_plane(z0 + 2, true);  // into the slot of phi(z0-3), no longer read
    prefetch_a(z0 - 1);
    cp_async_wait_all();
    __syncthreads();
    // theta partials of the first loop plane; the loop computes each later
    // plane's in the pull phase of the plane before
    theta_partials(z0);

    for (int q = z0 - 1; q <= z1; ++q) {
        bool zok = true;
        const int wz = zwrap(q, zok);
        const int zoff = wz * plane;
        const bool q_inner = (q >= z0) && (q < z1);

        // ================= phase 1 =================
        // partials of phi(q+3), then theta(q+2) from the partials of planes
        // q+1..q+3 (this thread's own nodes)
        planar_plane(q + 3);
        theta_plane(q + 2);

        R c4m = R(0), c40 = R(0), c4p = R(0);  // centre group of the interior node
        // unrolled: the interior node's copy of the collision reads the
        // prefetched registers in place (one shared copy of the loop body
        // costs moves and selects between the two sources: 6 % more
        // instructions and 3.6 % more time on the FP32 Laplace step)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int node = k ? nodeB : nodeA;
            if (node < 0) continue;
            const bool inb = zok && (k ? okB : okA);
            const int gi = zoff + (k ? offB : offA);
            NodeRaw cur;
            if (k == 0) cur = nxt;
            else if (inb) fetch(gi, cur);
            int isf = 1;
            if (inb && obs) isf = cur.isf;
            const bool live = inb && (isf != 0);
            const bool interior = (k == 0) && out_ok && q_inner;
            // the wall links of the interior node, loaded before its collision uses them
            unsigned links = 0;
            bool any_wall = false;
            if (k == 0 && obs) links = wall_links(p, interior && isf == -1, cur.row, tx, any_wall);
            R fpop[27];
            bool ring_done = false;  // a ring node's populations are stored already
            R sP = 0, spxx = 0, spyy = 0, spzz = 0, spxy = 0, spxz = 0, spyz = 0, som = 0;
            if (live) {
                R P, u, v, w, pxx, pyy, pzz, pxy, pxz, pyz;
                if constexpr (LY::split) {
                    P = (R)cur.v32[0]; u = (R)cur.v32[1]; v = (R)cur.v32[2]; w = (R)cur.v32[3];
                } else {
                    P = CD::dec(cur.m[0], p.inv_scale[0]);
                    u = CD::dec(cur.m[1], p.inv_scale[1]);
                    v = CD::dec(cur.m[2], p.inv_scale[2]);
                    w = CD::dec(cur.m[3], p.inv_scale[3]);
                }
                pxx = CD::dec(cur.m[4], p.inv_scale[4]);
                pyy = CD::dec(cur.m[5], p.inv_scale[5]);
                pzz = CD::dec(cur.m[6], p.inv_scale[6]);
                pxy = CD::dec(cur.m[7], p.inv_scale[7]);
                pxz = CD::dec(cur.m[8], p.inv_scale[8]);
                pyz = CD::dec(cur.m[9], p.inv_scale[9]);
                if constexpr (CD::scaled) {
                    // 16-bit storage keeps Pi - u u, the deviation from equilibrium
                    pxx += u * u; pyy += v * v; pzz += w * w;
                    pxy += u * v; pxz += u * w; pyz += v * w;
                }
                R phi = 0, lap = 0, divt = 0, gfx = 0, gfy = 0, gfz = 0;
                R phi_u = 0;         // phi before the mass correction
                bool stale = false;  // the collision reads phi_u (see below)
                const int hx = node % R1X, hy = node / R1X;
                const int c2 = (hy + 1) * R2X + (hx + 1);
                const int c3 = (hy + 2) * R3X + (hx + 2);
                phi = phis[phi_slot(q) * R3N + c3];
                const R phm = phis[phi_slot(q - 1) * R3N + c3], php = phis[phi_slot(q + 1) * R3N + c3];
                const R* sm = sxys + sxy_slot(q - 1) * R2N;
                const R* s0 = sxys + sxy_slot(q) * R2N;
                const R* sp = sxys + sxy_slot(q + 1) * R2N;
                // S_z S_x S_y phi - phi, with W0 - 1 = -2 W1
                lap = R(6) * (W1 * (sm[c2] + sp[c2]) + W0 * s0[c2] + W1 * ((phm - phi) + (php - phi)));
                const R* hm = hs + h_slot(q - 1) * (3 * R1N);
                const R* h0 = hs + h_slot(q) * (3 * R1N);
                const R* hp = hs + h_slot(q + 1) * (3 * R1N);
                divt = R(3) * ((W1 * (hm[node] + hp[node]) + W0 * h0[node]) +
                               W1 * ((hp[R1N + node] - hm[R1N + node]) + (hp[2 * R1N + node] - hm[2 * R1N + node])));
                const R* g1 = gts + gt_slot(q) * (3 * R1N);
                gfx = g1[0 * R1N + node];
                gfy = g1[1 * R1N + node];
                gfz = g1[2 * R1N + node];
                if constexpr (OBS) {
                    // from here on the input phi after the mass correction (the
                    // gradient, theta and Laplacian above are compute_norm's, from
                    // the uncorrected phi)
                    if (do_mcorr) {
                        phi_u = phi;
                        phi = (R)mass_corrected<SP>((double)phi, mcorr);
                        // a node reached across a periodic face is, in the
                        // reference's fused kernel, a halo copy: its moments and
                        // forces were exchanged after the moments kernel (corrected
                        // phi), its phi before the correction
                        stale = phi != phi_u && ((k ? wrapB : wrapA) || q < 0 || q >= nz);
                    }
                }
                // ---- moments prologue: lb_cuda_moments_module.f90:104-339 ----
                R inv = R(1), mask = R(0), fxv, fyv, fzv;
                mask = R(4) * phi * (R(1) - phi);
                if (dr) {
                    const R rhophi = p.rho_r * phi + (R(1) - phi) * p.rho_b;
                    inv = rcp<R>(rhophi);
                    fxv = rhophi * p.fx; fyv = rhophi * p.fy; fzv = rhophi * p.fz;
                } else {
                    fxv = p.fx; fyv = p.fy; fzv = p.fz;
                }
                R grx = 0, gry = 0, grz = 0, cv = 0, omega;
                R visc_l = p.visc1;  // local viscosity (mixture with two components)
                const R chem = R(4) * p.beta * phi * (phi - R(1)) * (phi - R(0.5)) - p.kapp * lap;
                fxv += chem * gfx;
                fyv += chem * gfy;
                fzv += chem * gfz;
                if constexpr (REP) {
                    // REPULSIVE_FLUX (lb_cuda_moments_module.f90:148-160): rho_phi F_rep,
                    // each component capped at 1e-3, times rho_phi
                    const R rh = dr ? p.rho_r * phi + (R(1) - phi) * p.rho_b : R(1);
                    const R cap = R(1.0e-3);
                    R t0 = p.rep[gi] * rh, t1 = p.rep[N + gi] * rh, t2 = p.rep[2 * N + gi] * rh;
                    t0 = t0 > cap ? cap : (t0 < -cap ? -cap : t0);
                    t1 = t1 > cap ? cap : (t1 < -cap ? -cap : t1);
                    t2 = t2 > cap ? cap : (t2 < -cap ? -cap : t2);
                    fxv += t0 * rh;
                    fyv += t1 * rh;
                    fzv += t2 * rh;
                }
                if (dr) {
                    const R drho = p.rho_r - p.rho_b;
                    grx = drho * gfx; gry = drho * gfy; grz = drho * gfz;
                    const R mp = mask * P * cssq;
                    fxv -= mp * grx; fyv -= mp * gry; fzv -= mp * grz;
                }
                R tfx = fxv, tfy = fyv, tfz = fzv;
                if (dr) {
                    const R uo = CD::dec(cur.uo[0], p.inv_scale[F_UOLD + 0]);
                    const R vo = CD::dec(cur.uo[1], p.inv_scale[F_UOLD + 1]);
                    const R wo = CD::dec(cur.uo[2], p.inv_scale[F_UOLD + 2]);
                    const R qxx = pxx - uo * uo, qyy = pyy - vo * vo, qzz = pzz - wo * wo;
                    const R qxy = pxy - uo * vo, qxz = pxz - uo * wo, qyz = pyz - vo * wo;
                    const R visc = (p.rho_r * p.visc1 * phi + (R(1) - phi) * p.visc2 * p.rho_b) * inv;
                    visc_l = visc;
                    omega = rcp<R>(visc * R(3) + R(0.5));
                    // mask * visc / (tau cs^2), with 1/tau = omega
                    cv = mask * visc * omega * R(3);
                    fxv -= cv * (qxx * grx + qxy * gry + qxz * grz);
                    fyv -= cv * (qyy * gry + qxy * grx + qyz * grz);
                    fzv -= cv * (qzz * grz + qxz * grx + qyz * gry);
                    const R tmp = -p.sharp_c * divt;
                    u += R(0.5) * fxv * inv;
                    v += R(0.5) * fyv * inv;
                    w += R(0.5) * fzv * inv;
                    const R dd = (p.rho_r - p.rho_b) * (p.tau_diff * lap + tmp);
                    const R den = rcp<R>(R(1) - R(0.5) * dd * inv);
                    u *= den; v *= den; w *= den;
                    tfx -= dd * u; tfy -= dd * v; tfz -= dd * w;
                    fxv -= dd * u; fyv -= dd * v; fzv -= dd * w;
                } else {
                    u += R(0.5) * fxv * inv;
                    v += R(0.5) * fyv * inv;
                    w += R(0.5) * fzv * inv;
                    const R visc = (p.rho_r * p.visc1 * phi + (R(1) - phi) * p.visc2 * p.rho_b) * inv;
                    visc_l = visc;
                    omega = rcp<R>(visc * R(3) + R(0.5));
                }
                pxx += fxv * u * inv;
                pyy += fyv * v * inv;
                pzz += fzv * w * inv;
                pxy += R(0.5) * (fyv * u + fxv * v) * inv;
                pxz += R(0.5) * (fzv * u + fxv * w) * inv;
                pyz += R(0.5) * (fzv * v + fyv * w) * inv;
                if (dr) {
                    const R qxx = pxx - u * u, qyy = pyy - v * v, qzz = pzz - w * w;
                    const R qxy = pxy - u * v, qxz = pxz - u * w, qyz = pyz - v * w;
                    tfx -= cv * (qxx * grx + qxy * gry + qxz * grz);
                    tfy -= cv * (qyy * gry + qxy * grx + qyz * grz);
                    tfz -= cv * (qzz * grz + qxz * grx + qyz * gry);
                }
                // ---- outputs of this node that leave the kernel ----
                if (interior) {
                    if (p.write_u) {
                        CD::st(p.uout + 0 * N, gi, u, p.scale[F_UOLD + 0]);
                        CD::st(p.uout + 1 * N, gi, v, p.scale[F_UOLD + 1]);
                        CD::st(p.uout + 2 * N, gi, w, p.scale[F_UOLD + 2]);
                    }
                    // update_phifields: lb_cuda_update_phi_module.f90:77-93
                    const R phi_new = phi - u * R(0.5) * gfx - v * R(0.5) * gfy - w * R(0.5) * gfz +
                                      p.tau_diff * lap - p.sharp_c * divt;
                    CP::st(p.pout, gi, phi_new, p.scale[F_PHI]);
                }
                if constexpr (OBS) {
                    if (stale) {
                        // density and viscosity of the collision from the halo copy's
                        // uncorrected phi (lb_cuda_fused_module.f90:590-620)
                        const R rh = dr ? p.rho_r * phi_u + (R(1) - phi_u) * p.rho_b : R(1);
                        if (dr) inv = rcp<R>(rh);
                        visc_l = (p.rho_r * p.visc1 * phi_u + (R(1) - phi_u) * p.visc2 * p.rho_b) * inv;
                        omega = rcp<R>(visc_l * R(3) + R(0.5));
                    }
                }
                // ---- collision: lb_cuda_fused_module.f90:531-713 ----
                const R Xn = pxx - u * u, Yn = pyy - v * v, Zn = pzz - w * w;
                const R XYn = pxy - u * v, XZn = pxz - u * w, YZn = pyz - v * w;
                const R Fx = tfx * inv, Fy = tfy * inv, Fz = tfz * inv;
                if (p.smag) {
                    // SMAGORINSKI (lb_cuda_fused_module.f90:609-616): relaxation time from the
                    // Frobenius norm of the non-equilibrium stress; the moments prologue above
                    // keeps the molecular one, as the reference's moments kernel does
                    const R QQ = Xn * Xn + Yn * Yn + Zn * Zn + R(2) * (XYn * XYn + XZn * XZn + YZn * YZn);
                    const R v3 = R(3) * visc_l;
                    const R tau = R(0.5) + R(1.0 / 6.0) * (v3 + sqrt_a<R>(v3 * v3 + R(SMAG_C) * sqrt_a<R>(R(2) * QQ) * inv));
                    omega = rcp<R>(tau);
                }
                sP = P;
                spxx = Xn; spyy = Yn; spzz = Zn; spxy = XYn; spxz = XZn; spyz = YZn; som = omega;
                const R om1 = R(1) - omega;
                const R m0 = P;
                const R mx = u + R(0.5) * Fx, my = v + R(0.5) * Fy, mz = w + R(0.5) * Fz;
                const R mxx = u * u + om1 * Xn + u * Fx;
                const R myy = v * v + om1 * Yn + v * Fy;
                const R mzz = w * w + om1 * Zn + w * Fz;
                const R mxy = u * v + om1 * XYn + R(0.5) * (u * Fy + v * Fx);
                const R mxz = u * w + om1 * XZn + R(0.5) * (u * Fz + w * Fx);
                const R myz = v * w + om1 * YZn + R(0.5) * (v * Fz + w * Fy);
                if constexpr (LAT == 27) {
                    R M[3][3][3];
                    M[0][0][0] = m0;
                    M[1][0][0] = mx; M[0][1][0] = my; M[0][0][1] = mz;
                    M[2][0][0] = mxx; M[0][2][0] = myy; M[0][0][2] = mzz;
                    M[1][1][0] = mxy; M[1][0][1] = mxz; M[0][1][1] = myz;
                    if constexpr (HO) {
                        if constexpr (OBS == 1) ho_rows<R>(M, u, v, w, om1, Xn, Yn, Zn, XYn, XZn, YZn);
                        else ho_rows_wide<R>(M, u, v, w, om1, Xn, Yn, Zn, XYn, XZn, YZn);
                    } else {
                        M[2][1][0] = M[2][0][1] = M[1][2][0] = M[1][0][2] = M[0][1][2] = M[0][2][1] = M[1][1][1] = R(0);
                        M[2][2][0] = M[2][0][2] = M[0][2][2] = M[1][1][2] = M[1][2][1] = M[2][1][1] = R(0);
                        M[2][1][2] = M[2][2][1] = M[1][2][2] = M[2][2][2] = R(0);
                    }
                    if (k == 0) {
                        full_pops27<R>(M, fpop);
                    } else {
                        // a ring node's populations go to shared memory at once
                        const bool plus = ring_dir > R(0);
                        if (ring_col)
                            ring_col_pops27<R>(M, ring_dir, [&](int b, R vm, R v0, R vp) {
                                put_group(3 * b + (plus ? 2 : 0), node, vm, v0, vp);
                            });
                        else
                            ring_row_pops27<R>(M, ring_dir, [&](int a, R vm, R v0, R vp) {
                                put_group(3 * (plus ? 2 : 0) + a, node, vm, v0, vp);
                            });
                        ring_done = true;
                    }
                } else {
                    low_order_pops<LAT, R>(m0, mx, my, mz, mxx, myy, mzz, mxy, mxz, myz, fpop);
                }
            } else {
#pragma unroll
                for (int l = 0; l < 27; ++l) fpop[l] = R(0);
            }
#pragma unroll
            for (int g = 0; g < 9; ++g) {
                if (ring_done) break;
                const int cx = g % 3 - 1, cy = g / 3 - 1;
                // links the lattice lacks carry 0 (D3Q19: no corners, D3Q15: no edges)
                R2 v;
                v.x = IN<LAT>(LINK(cx, cy, -1)) ? fpop[LINK(cx, cy, -1)] : R(0);
                v.y = IN<LAT>(LINK(cx, cy, 0)) ? fpop[LINK(cx, cy, 0)] : R(0);
                const R vp = IN<LAT>(LINK(cx, cy, 1)) ? fpop[LINK(cx, cy, 1)] : R(0);
                if (g == 4) {
                    // the centre group: only the interior node's own output reads it
                    if (k == 0) {
                        c4m = v.x;
                        c40 = v.y;
                        c4p = vp;
                    }
                    continue;
                }
                pops2[gslot(g) * R1N + node] = v;
                pops1[gslot(g) * R1N + node] = vp;
            }

            // ---- obstacle bounce-back: lb_cuda_boundary_module.f90:162-199 ----
            if (k == 0 && any_wall) {
                R d[10];
                wall_link_sums<LAT, R>(links, sP, R(1) - som, spxx, spyy, spzz, spxy, spxz, spyz, d);
#pragma unroll
                for (int i = 0; i < 10; ++i) A2[i].y += d[i];
            }
        }
        // the interior node's fields of plane q+1, issued before the barrier
        // rather than after it: 0.9 % per step at 256^3
        prefetch_a(q + 1);
        __syncthreads();

        // ================= phase 2 =================
        // the slot of phi(q-1) was last read in phase 1
        load_phi_plane(q + 4, true);
        if (obs) theta_isf(q + 3, th_isf);  // for theta(q+3), next plane
        // the theta partials of plane q+2 at this thread's collision nodes
        // (theta(q+2) is complete since the barrier after phase 1).  Here
        // rather than in phase 1 they fill the shorter pull phase and shorten
        // the collision phase, whose barrier waits for the ring collisions
        // (1.7 % per step at 256^3); before the pull rather than after it,
        // 0.3 % more
        theta_partials(q + 2);

        // the three cz populations of every (cx, cy) group from node x - c:
        // cz = -1, 0 as one pair (packed sums), cz = +1 alone
        using PP = typename PK<R>::T;
        PP gp[3][3];  // [cy][cx]
        R gs[3][3];
#pragma unroll
        for (int yc = 0; yc < 3; ++yc)
#pragma unroll
            for (int xc = 0; xc < 3; ++xc) {
                const int g = 3 * yc + xc;
                if (g == 4) {
                    gp[yc][xc] = PK<R>::mk(c4m, c40);
                    gs[yc][xc] = c4p;
                    continue;
                }
                const int src = (ty + 1 - (yc - 1)) * R1X + (tx + 1 - (xc - 1));
                const R2 v = pops2[gslot(g) * R1N + src];
                gp[yc][xc] = PK<R>::mk(v.x, v.y);
                gs[yc][xc] = pops1[gslot(g) * R1N + src];
            }
        pull_sums27<R>(gp, gs, A2, ap);
        R am[10];
#pragma unroll
        for (int i = 0; i < 10; ++i) am[i] = A2[i].x;
        if (q - 1 >= z0 && out_ok) write_moments<S, R>(p, (q - 1) * plane + out_off, am);
#pragma unroll
        for (int i = 0; i < 10; ++i) {
            A2[i] = PK<R>::mk(A2[i].y, ap[i]);
            ap[i] = R(0);
        }
        cp_async_wait_all();
        __syncthreads();
    }
}

// CTAs per SM the kernel is compiled for: two of 8-row tiles, one of 16 rows, one
// in FP64, and one of 8 rows of D3Q27 HIGHORDER with one component, whose
// two spill up to 264 bytes in 80 registers (FP32, a step of 200^3 in 16-plane
// segments 388 us with two, 365 us with one; of 40^3 21.3 and 13.9 us)
template <int LAT, bool HO, bool TC, typename R, int TYV> constexpr int step_min_blocks() {
    return (sizeof(R) == 8 || TYV > 8 || (LAT == 27 && HO && !TC)) ? 1 : 2;
}

// threads and shared memory of a CTA, by component class
template <bool TC, int TYV> constexpr int step_threads() { return TC ? TX * TYV : single_threads<TYV>(); }
template <int LAT, bool TC, typename S, typename R, int TYV> constexpr size_t step_smem_bytes() {
    if constexpr (TC) return stream_smem_bytes<S, R, TYV>();
    else return single_smem_bytes<LAT, R, TYV>();
}
template <int LAT, bool HO, bool TC, typename S, typename R, int TYV, bool REP, int OBS>
__device__ __forceinline__ void any_body(const StepParams<S, R>& p, int bx, int by, int z0, int z1) {
    if constexpr (TC) step_body<LAT, HO, S, R, TYV, REP, OBS>(p, bx, by, z0, z1);
    else single_body<LAT, HO, S, R, TYV, (OBS & 1) != 0>(p, bx, by, z0, z1);
}

// Column-planes of the planes zlo .. zlo + nzr - 1 of a box for a tile of
// TYV rows, column index = by * gx + bx, plane fastest.
template <int TYV, typename F>
__device__ __forceinline__ void run_share(const int nx, const int nzr, const int zlo, long long s0, long long s1,
                                          F&& body) {
    const int gx = (nx + TX - 1) / TX;
    while (s0 < s1) {
        const long long col = s0 / nzr;
        const int z0 = (int)(s0 - col * nzr);
        const int z1 = (int)min((long long)nzr, z0 + (s1 - s0));
        body((int)(col % gx), (int)(col / gx), zlo + z0, zlo + z1);
        s0 += z1 - z0;
    }
}

// Single box.  zseg > 0: one CTA per (tile x, tile y, z segment of zseg
// planes).  zseg < 0: split columns -- CTA i < ncols advances planes [0, L)
// of column i and CTA ncols + i planes [L, nzr), L = -zseg: when the columns
// fill less than one wave of CTA slots, the long segments run in step on
// ncols SMs (their halo re-reads hit in L2) while the other SMs work through
// the short tails.  zseg = 0: persistent schedule -- the box's columns x planes are
// cut into gridDim.x equal contiguous shares (a share may end inside one
// column and continue at the bottom of the next), so every CTA does the same
// work and pays the pipeline fill of a segment start only once or twice.
// Both schedules are expressed as a range of column-planes walked by ONE call
// site of step_body, so the kernel holds a single compiled copy of the step:
// separately inlined copies may contract floating-point operations
// differently and give results that differ in the last bit.
template <int LAT, bool HO, bool TC, typename S, typename R, int TYV, bool REP = false, int OBS = 1>
__global__ void __launch_bounds__(step_threads<TC, TYV>(), step_min_blocks<LAT, HO, TC, R, TYV>()) stream_kernel(const StepParams<S, R> p) {
    chain_begin();
    long long s0, s1;
    const int nzr = p.zhi - p.zlo;
    if (p.zseg < 0) {
        const int L = min(-p.zseg, nzr);
        const long long ncols = (long long)((p.nx + TX - 1) / TX) * ((p.ny + TYV - 1) / TYV);
        const bool head = blockIdx.x < ncols;
        const long long col = head ? blockIdx.x : blockIdx.x - ncols;
        s0 = col * nzr + (head ? 0 : L);
        s1 = col * nzr + (head ? L : nzr);
    } else if (p.zseg > 0) {
        const long long col = (long long)blockIdx.y * ((p.nx + TX - 1) / TX) + blockIdx.x;
        const int z0 = blockIdx.z * p.zseg;
        s0 = col * nzr + z0;
        s1 = s0 + min(p.zseg, nzr - z0);
    } else {
        const long long W = (long long)((p.nx + TX - 1) / TX) * ((p.ny + TYV - 1) / TYV) * nzr;
        const long long share = (W + gridDim.x - 1) / gridDim.x;
        s0 = (long long)blockIdx.x * share;
        s1 = min(W, s0 + share);
    }
    run_share<TYV>(p.nx, nzr, p.zlo, s0, s1,
                   [&](int bx, int by, int z0, int z1) { any_body<LAT, HO, TC, S, R, TYV, REP, OBS>(p, bx, by, z0, z1); });
}

// Many boxes in one launch: CTA i advances box work[i].x over column-planes
// [work[i].y, work[i].z) of that box (column-major: plane fastest), with the
// box's own parameters and fields.  A box gives the same bits whatever else is
// in the batch.  Each node's operations are those of stream_kernel, but in
// another compilation, where the compiler contracts the products of the
// two-component collision differently: the two agree to rounding.
template <int LAT, bool HO, bool TC, typename S, typename R, int TYV, bool REP = false, int OBS = 1>
__global__ void __launch_bounds__(step_threads<TC, TYV>(), step_min_blocks<LAT, HO, TC, R, TYV>())
    stream_kernel_batched(const StepParams<S, R>* __restrict__ boxes, const int4* __restrict__ work) {
    __shared__ StepParams<S, R> sp;
    chain_begin();
    const int4 w = work[blockIdx.x];
    if (threadIdx.x == 0) sp = boxes[w.x];
    __syncthreads();
    run_share<TYV>(sp.nx, sp.nz, 0, w.y, w.z,
                   [&](int bx, int by, int z0, int z1) { any_body<LAT, HO, TC, S, R, TYV, REP, OBS>(sp, bx, by, z0, z1); });
}

}  // namespace lbf
