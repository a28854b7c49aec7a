// lbf_single_kernel.cuh -- body of the fused step kernel for one component.
//
// Without the phase-field stencils a plane is a collision and a pull, so the
// work is laid out for those alone:
//  * every collision of the tile + 1-node ring has a thread of its own -- one
//    warp per tile row and RW warps for the ring -- so no warp carries two;
//  * the populations alternate between two shared buffers, so a plane has one
//    barrier: the pull of plane q and the collision of plane q+1 run without
//    one between them;
//  * every node's fields, the ring's too, are loaded one plane ahead;
//  * links that the lattice lacks are neither stored nor summed, and D3Q19 /
//    D3Q15 populations are built in opposite pairs.
// The sums go in the order of step_body, and the products of the collision are
// rounded as it rounds them, so the bits are those of the shared body of both
// component classes that this one replaced.
// Bound by issue and by the latency between a plane's barriers (20 warps, 0.6
// instructions a cycle and scheduler); registers hold it to one CTA of 16 rows
// or two of 8 (one with HIGHORDER).  FP32, 200 x 184 x 168, a step: D3Q19 265 us
// in the shared body, 154 us here; D3Q27 HIGHORDER with SMAGORINSKI 317 and 281 us
// (267 us with the sums of the rows and populations regrouped, which rounds
// differently).  D3Q27 does not fit in the 96 registers of 16 rows (FP32 spills
// 32-36 bytes, 104-136 with obstacles) nor, without HIGHORDER, in the 80 of 8
// rows (92 and 216 bytes); FP64, with 168, spills up to 204.
#pragma once
#include "lbf_node.cuh"

namespace lbf {

// Which populations of a (cx, cy) group g = 3 (cy + 1) + (cx + 1) a lattice
// has, and where they sit in shared memory: groups of three hold (cz = -1, 0)
// as a pair and +1 alone, groups of two (cz = -1, +1) a pair, groups of one
// (cz = 0) that one alone.  The centre group stays in registers.
// (Closed forms: as loops over the links these would be left to run time.)
template <int LAT> struct PopGroups {
    static __host__ __device__ constexpr bool corner(int g) { return g % 2 == 0 && g != 4; }
    static __host__ __device__ constexpr int count(int g) {
        return g == 4 || LAT == 27 ? 3 : LAT == 19 ? (corner(g) ? 1 : 3) : (corner(g) ? 2 : 1);
    }
    static __host__ __device__ constexpr int pair_slot(int g) {
        return LAT == 27 ? (g < 4 ? g : g - 1) : LAT == 19 ? g / 2 : (g < 4 ? g / 2 : g / 2 - 1);
    }
    static __host__ __device__ constexpr int single_slot(int g) { return LAT == 15 ? g / 2 : (g < 4 ? g : g - 1); }
    static constexpr int NPAIR = LAT == 27 ? 8 : 4, NSINGLE = LAT == 15 ? 4 : 8;
};

template <int LAT, typename R, int TYV> constexpr size_t single_smem_bytes() {
    return 2 * sizeof(R) * size_t(2 * PopGroups<LAT>::NPAIR + PopGroups<LAT>::NSINGLE) * Tile<TYV>::R1N;
}
// threads of a CTA: the tile's nodes and its ring, a whole number of warps each
template <int TYV> constexpr int single_threads() { return Tile<TYV>::NT + 32 * Tile<TYV>::RW; }

// A value that may be absent at compile time: sums of the links that a
// lattice has (a + 0 would not be dropped: it is not exact for a = -0)
template <typename R> struct Maybe {
    R v;
    bool has;
    __device__ __forceinline__ Maybe operator+(const Maybe& o) const {
        return has ? (o.has ? Maybe{v + o.v, true} : *this) : o;
    }
    __device__ __forceinline__ Maybe operator-(const Maybe& o) const {
        return has ? (o.has ? Maybe{v - o.v, true} : *this) : Maybe{-o.v, o.has};
    }
    __device__ __forceinline__ void add_to(R& a) const {
        if (has) a += v;
    }
    __device__ __forceinline__ void sub_from(R& a) const {
        if (has) a -= v;
    }
};

// One piece of a time step: tile (bx, by) of the box, planes z0 <= z < z1.
template <int LAT, bool HO, typename S, typename R, int TYV, bool OBS>
__device__ __forceinline__ void single_body(const StepParams<S, R>& p, const int bx, const int by, const int z0,
                                            const int z1) {
    using TL = Tile<TYV>;
    using PG = PopGroups<LAT>;
    using CD = Codec<S>;
    using LY = Layout<S>;
    using R2 = typename Vec2<R>::type;
    using PA = typename PK<R>::T;
    constexpr int TY = TL::TY, NT = TL::NT, R1Y = TL::R1Y, R1N = TL::R1N;
    constexpr int BUF = (2 * PG::NPAIR + PG::NSINGLE) * R1N;  // values of one buffer
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* const smem = reinterpret_cast<R*>(smem_raw);

    const int t = threadIdx.x;
    const bool inner = t < NT;  // uniform across a warp
    const int tx = t % TX, ty = t / TX;
    const int X0 = bx * TX, Y0 = by * TY;
    const long long N = p.N;
    const int plane = (int)p.plane;
    const int nx = p.nx, ny = p.ny, nz = p.nz;
    const bool obs = OBS && p.obstacles != 0;

    // this thread's collision node: a tile node, or a ring node -- the inner
    // 32 nodes of the top row, of the bottom row, then the left and right
    // columns with the corners.  Ring nodes stream into the tile along one
    // axis only: the rows' along y (cy = +1 from the top row, -1 from the
    // bottom), the columns' along x.
    const bool ring_col = t >= NT + 2 * TX;
    int hx = tx + 1, hy = ty + 1;
    bool have = true;
    if (!inner) {
        const int r = t - NT;
        if (!ring_col) {
            hx = r % TX + 1;
            hy = r < TX ? 0 : R1Y - 1;
        } else {
            const int c = r - 2 * TX;
            have = c < 2 * R1Y;
            hx = c < R1Y ? 0 : R1X - 1;
            hy = c < R1Y ? c : c - R1Y;
        }
    }
    const int node = hy * R1X + hx;
    const R dir = ring_col ? (hx == 0 ? R(1) : R(-1)) : (hy == 0 ? R(1) : R(-1));
    const bool plus = dir > R(0);
    bool ok = have;
    const int gx = wrap_coord(X0 + hx - 1, nx, p.pbx, ok);
    const int gy = wrap_coord(Y0 + hy - 1, ny, p.pby, ok);
    const int off = ok ? gy * nx + gx : 0;
    const bool out_ok = inner && X0 + tx < nx && Y0 + ty < ny;
    const int out_off = (Y0 + ty) * nx + X0 + tx;

    auto put = [&](R* buf, int g, R vm, R v0, R vp) {
        R2* const pairs = reinterpret_cast<R2*>(buf);
        R* const singles = buf + 2 * PG::NPAIR * R1N;
        const int n = PG::count(g);
        if (n == 3) {
            R2 v;
            v.x = vm;
            v.y = v0;
            pairs[PG::pair_slot(g) * R1N + node] = v;
            singles[PG::single_slot(g) * R1N + node] = vp;
        } else if (n == 2) {
            R2 v;
            v.x = vm;
            v.y = vp;
            pairs[PG::pair_slot(g) * R1N + node] = v;
        } else {
            singles[PG::single_slot(g) * R1N + node] = v0;
        }
    };

    // this node's stored moments (and isfluid) of the next plane, not yet decoded
    struct NodeRaw {
        S m[10];       // with 16-bit storage only m[4..9] (Pi - u u)
        float v32[4];  // P, u, v, w of the 16-bit formats
        int8_t isf;
        int row;       // start of the warp's wall links
    } nxt;
    auto prefetch = [&](int q) {
        bool zk = true;
        const int wz = wrap_coord(q, nz, p.pbz, zk);
        if (!(zk && ok)) return;
        const int gi = wz * plane + off;
        if constexpr (LY::split) {
#pragma unroll
            for (int f = 0; f < 4; ++f) nxt.v32[f] = p.pres_in[f * N + gi];
#pragma unroll
            for (int f = 4; f < 10; ++f) nxt.m[f] = CD::raw(p.min + LY::off(f, N), gi);
        } else {
#pragma unroll
            for (int f = 0; f < 10; ++f) nxt.m[f] = CD::raw(p.min + f * N, gi);
        }
        if (obs) nxt.isf = p.isf[gi];
    };
    const int segs = (nx + TX - 1) / TX;
    auto prefetch_row = [&](int q) {
        if (obs && inner && q >= z0 && q < z1 && Y0 + ty < ny) nxt.row = __ldg(p.link_rows + (q * ny + Y0 + ty) * segs + bx);
    };

    // raw moments {sum g, sum g c, sum g c c} of output planes q-1, q as pairs, and q+1
    PA A2[10];
    R ap[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        A2[i] = PK<R>::mk(R(0), R(0));
        ap[i] = R(0);
    }
    // a CTA that walks several pieces starts the next one when its last pull is done
    __syncthreads();
    prefetch(z0 - 1);
    nxt.row = 0;
    int b = 0;
    for (int q = z0 - 1; q <= z1; ++q, b ^= 1) {
        R* const buf = smem + b * BUF;
        bool zok = true;
        const int wz = wrap_coord(q, nz, p.pbz, zok);
        const bool inb = zok && ok;
        const int gi = wz * plane + off;
        const int isf = obs && inb ? nxt.isf : 1;
        R c4m = R(0), c40 = R(0), c4p = R(0);  // centre group
        const bool interior = out_ok && inb && q >= z0 && q < z1;
        unsigned links = 0;
        bool any_wall = false;
        if (obs && inner) links = wall_links(p, interior && isf == -1, nxt.row, tx, any_wall);
        if (inb && isf != 0) {
            R P, u, v, w;
            if constexpr (LY::split) {
                P = (R)nxt.v32[0]; u = (R)nxt.v32[1]; v = (R)nxt.v32[2]; w = (R)nxt.v32[3];
            } else {
                P = CD::dec(nxt.m[0], p.inv_scale[0]);
                u = CD::dec(nxt.m[1], p.inv_scale[1]);
                v = CD::dec(nxt.m[2], p.inv_scale[2]);
                w = CD::dec(nxt.m[3], p.inv_scale[3]);
            }
            R pxx = CD::dec(nxt.m[4], p.inv_scale[4]), pyy = CD::dec(nxt.m[5], p.inv_scale[5]);
            R pzz = CD::dec(nxt.m[6], p.inv_scale[6]), pxy = CD::dec(nxt.m[7], p.inv_scale[7]);
            R pxz = CD::dec(nxt.m[8], p.inv_scale[8]), pyz = CD::dec(nxt.m[9], p.inv_scale[9]);
            if constexpr (CD::scaled) {
                // 16-bit storage keeps Pi - u u, the deviation from equilibrium
                pxx = fmaf_t(u, u, pxx); pyy = fmaf_t(v, v, pyy); pzz = fmaf_t(w, w, pzz);
                pxy = fmaf_t(u, v, pxy); pxz = fmaf_t(u, w, pxz); pyz = fmaf_t(v, w, pyz);
            }
            // ---- moments prologue: lb_cuda_moments_module.f90:104-339 ----
            const R Fx = p.fx, Fy = p.fy, Fz = p.fz;
            u += R(0.5) * Fx;
            v += R(0.5) * Fy;
            w += R(0.5) * Fz;
            pxx += Fx * u;
            pyy += Fy * v;
            pzz += Fz * w;
            pxy += R(0.5) * (Fy * u + Fx * v);
            pxz += R(0.5) * (Fz * u + Fx * w);
            pyz += R(0.5) * (Fz * v + Fy * w);
            if (interior && p.write_u) {
                CD::st(p.uout + 0 * N, gi, u, p.scale[F_UOLD + 0]);
                CD::st(p.uout + 1 * N, gi, v, p.scale[F_UOLD + 1]);
                CD::st(p.uout + 2 * N, gi, w, p.scale[F_UOLD + 2]);
            }
            // ---- collision: lb_cuda_fused_module.f90:531-713 ----
            const R uu = mul_rn(u, u), vv = mul_rn(v, v), ww = mul_rn(w, w);
            const R uv = mul_rn(u, v), uw = mul_rn(u, w), vw = mul_rn(v, w);
            const R Xn = pxx - uu, Yn = pyy - vv, Zn = pzz - ww;
            const R XYn = pxy - uv, XZn = pxz - uw, YZn = pyz - vw;
            R omega = p.omega;
            if (p.smag) {
                // SMAGORINSKI (lb_cuda_fused_module.f90:609-616)
                const R q1 = fmaf_t(Zn, Zn, fmaf_t(Xn, Xn, mul_rn(Yn, Yn)));
                const R q2 = fmaf_t(YZn, YZn, fmaf_t(XYn, XYn, mul_rn(XZn, XZn)));
                const R QQ = fmaf_t(R(2), q2, q1);
                const R v3 = R(3) * p.visc1;
                const R tau = fmaf_t(R(1.0 / 6.0), v3 + sqrt_a<R>(fmaf_t(v3, v3, mul_rn(R(SMAG_C), sqrt_a<R>(R(2) * QQ)))), R(0.5));
                omega = rcp<R>(tau);
            }
            const R om1 = R(1) - omega;
            const R mx = u + R(0.5) * Fx, my = v + R(0.5) * Fy, mz = w + R(0.5) * Fz;
            const R mxx = fmaf_t(u, Fx, fmaf_t(om1, Xn, uu));
            const R myy = fmaf_t(v, Fy, fmaf_t(om1, Yn, vv));
            const R mzz = fmaf_t(w, Fz, fmaf_t(om1, Zn, ww));
            const R mxy = fmaf_t(R(0.5), u * Fy + v * Fx, fmaf_t(om1, XYn, uv));
            const R mxz = fmaf_t(R(0.5), u * Fz + w * Fx, fmaf_t(om1, XZn, uw));
            const R myz = fmaf_t(R(0.5), v * Fz + w * Fy, fmaf_t(om1, YZn, vw));
            R fpop[27];
            if constexpr (LAT == 27) {
                R M[3][3][3];
                M[0][0][0] = P;
                M[1][0][0] = mx; M[0][1][0] = my; M[0][0][1] = mz;
                M[2][0][0] = mxx; M[0][2][0] = myy; M[0][0][2] = mzz;
                M[1][1][0] = mxy; M[1][0][1] = mxz; M[0][1][1] = myz;
                if constexpr (HO) {
                    ho_rows_wide<R>(M, u, v, w, om1, Xn, Yn, Zn, XYn, XZn, YZn);
                } else {
                    M[2][1][0] = M[2][0][1] = M[1][2][0] = M[1][0][2] = M[0][1][2] = M[0][2][1] = M[1][1][1] = R(0);
                    M[2][2][0] = M[2][0][2] = M[0][2][2] = M[1][1][2] = M[1][2][1] = M[2][1][1] = R(0);
                    M[2][1][2] = M[2][2][1] = M[1][2][2] = M[2][2][2] = R(0);
                }
                if (inner)
                    full_pops27<R>(M, fpop);
                else if (ring_col)
                    ring_col_pops27<R>(M, dir, [&](int k, R vm, R v0, R vp) {
                        put(buf, 3 * k + (plus ? 2 : 0), vm, v0, vp);
                    });
                else
                    ring_row_pops27<R>(M, dir, [&](int k, R vm, R v0, R vp) {
                        put(buf, 3 * (plus ? 2 : 0) + k, vm, v0, vp);
                    });
            } else {
                low_order_pops<LAT, R>(P, mx, my, mz, mxx, myy, mzz, mxy, mxz, myz, fpop);
                if (!inner) {
                    // the three groups of this ring node that enter the tile:
                    // the value of either direction goes to its own slot
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        if (ring_col) {
                            if (plus) put(buf, 3 * k + 2, fpop_or0<LAT>(fpop, LINK(1, k - 1, -1)), fpop_or0<LAT>(fpop, LINK(1, k - 1, 0)), fpop_or0<LAT>(fpop, LINK(1, k - 1, 1)));
                            else put(buf, 3 * k, fpop_or0<LAT>(fpop, LINK(-1, k - 1, -1)), fpop_or0<LAT>(fpop, LINK(-1, k - 1, 0)), fpop_or0<LAT>(fpop, LINK(-1, k - 1, 1)));
                        } else {
                            if (plus) put(buf, 6 + k, fpop_or0<LAT>(fpop, LINK(k - 1, 1, -1)), fpop_or0<LAT>(fpop, LINK(k - 1, 1, 0)), fpop_or0<LAT>(fpop, LINK(k - 1, 1, 1)));
                            else put(buf, k, fpop_or0<LAT>(fpop, LINK(k - 1, -1, -1)), fpop_or0<LAT>(fpop, LINK(k - 1, -1, 0)), fpop_or0<LAT>(fpop, LINK(k - 1, -1, 1)));
                        }
                    }
                }
            }
            if (inner) {
#pragma unroll
                for (int g = 0; g < 9; ++g) {
                    if (g == 4) continue;
                    const int cx = g % 3 - 1, cy = g / 3 - 1;
                    put(buf, g, fpop_or0<LAT>(fpop, LINK(cx, cy, -1)), fpop_or0<LAT>(fpop, LINK(cx, cy, 0)), fpop_or0<LAT>(fpop, LINK(cx, cy, 1)));
                }
                c4m = fpop_or0<LAT>(fpop, LINK(0, 0, -1));
                c40 = fpop[0];
                c4p = fpop_or0<LAT>(fpop, LINK(0, 0, 1));
            }
            if constexpr (OBS) {
                // ---- obstacle bounce-back: lb_cuda_boundary_module.f90:162-199 ----
                if (any_wall) {
                    R d[10];
                    wall_link_sums<LAT, R>(links, P, om1, Xn, Yn, Zn, XYn, XZn, YZn, d);
#pragma unroll
                    for (int i = 0; i < 10; ++i) A2[i].y += d[i];
                }
            }
        } else if (have) {
            // a solid node or one outside the box sends nothing
#pragma unroll
            for (int g = 0; g < 9; ++g)
                if (g != 4) put(buf, g, R(0), R(0), R(0));
        }
        // the next plane's fields: their latency passes behind the barrier and the pull
        prefetch(q + 1);
        prefetch_row(q + 1);
        __syncthreads();
        if (!inner) continue;

        // the populations of every (cx, cy) group from node x - c
        const R2* const pairs = reinterpret_cast<const R2*>(buf);
        const R* const singles = buf + 2 * PG::NPAIR * R1N;
        if constexpr (LAT == 27) {
            using P = PK<R>;
            PA gp[3][3];  // [cy][cx], (cz = -1, 0)
            R gs[3][3];   // cz = +1
#pragma unroll
            for (int yc = 0; yc < 3; ++yc)
#pragma unroll
                for (int xc = 0; xc < 3; ++xc) {
                    const int g = 3 * yc + xc;
                    if (g == 4) {
                        gp[yc][xc] = P::mk(c4m, c40);
                        gs[yc][xc] = c4p;
                        continue;
                    }
                    const int src = node - (yc - 1) * R1X - (xc - 1);
                    const R2 v = pairs[PG::pair_slot(g) * R1N + src];
                    gp[yc][xc] = P::mk(v.x, v.y);
                    gs[yc][xc] = singles[PG::single_slot(g) * R1N + src];
                }
            pull_sums27<R>(gp, gs, A2, ap);
        } else {
#pragma unroll
            for (int cz = -1; cz <= 1; ++cz) {
                Maybe<R> f[3][3];  // [cy][cx]
#pragma unroll
                for (int g = 0; g < 9; ++g) {
                    const int cx = g % 3 - 1, cy = g / 3 - 1;
                    Maybe<R>& h = f[g / 3][g % 3];
                    h.has = IN<LAT>(LINK(cx, cy, cz));
                    if (!h.has) continue;
                    const int src = node - cy * R1X - cx;
                    if (g == 4) h.v = cz < 0 ? c4m : cz == 0 ? c40 : c4p;
                    else if (PG::count(g) == 3 && cz < 1) h.v = cz < 0 ? pairs[PG::pair_slot(g) * R1N + src].x : pairs[PG::pair_slot(g) * R1N + src].y;
                    else if (PG::count(g) == 2) h.v = cz < 0 ? pairs[PG::pair_slot(g) * R1N + src].x : pairs[PG::pair_slot(g) * R1N + src].y;
                    else h.v = singles[PG::single_slot(g) * R1N + src];
                }
                // the sums of pull_sums27, in its order
                Maybe<R> S0[3], S1[3], S2[3];
#pragma unroll
                for (int y = 0; y < 3; ++y) {
                    S0[y] = (f[y][0] + f[y][1]) + f[y][2];
                    S1[y] = f[y][2] - f[y][0];
                    S2[y] = f[y][2] + f[y][0];
                }
                const Maybe<R> Y00 = (S0[0] + S0[1]) + S0[2], Y01 = S0[2] - S0[0], Y02 = S0[2] + S0[0];
                const Maybe<R> Y10 = (S1[0] + S1[1]) + S1[2], Y11 = S1[2] - S1[0], Y20 = (S2[0] + S2[1]) + S2[2];
                R a[10];
#pragma unroll
                for (int i = 0; i < 10; ++i) a[i] = cz < 0 ? A2[i].x : cz == 0 ? A2[i].y : ap[i];
                Y00.add_to(a[0]);
                Y10.add_to(a[1]);
                Y01.add_to(a[2]);
                Y20.add_to(a[4]);
                Y02.add_to(a[5]);
                Y11.add_to(a[7]);
                if (cz) {
                    Y00.add_to(a[6]);
                    if (cz > 0) { Y00.add_to(a[3]); Y10.add_to(a[8]); Y01.add_to(a[9]); }
                    else { Y00.sub_from(a[3]); Y10.sub_from(a[8]); Y01.sub_from(a[9]); }
                }
#pragma unroll
                for (int i = 0; i < 10; ++i) {
                    if (cz < 0) A2[i].x = a[i];
                    else if (cz == 0) A2[i].y = a[i];
                    else ap[i] = a[i];
                }
            }
        }
        R am[10];
#pragma unroll
        for (int i = 0; i < 10; ++i) am[i] = A2[i].x;
        if (q - 1 >= z0 && out_ok) write_moments<S, R>(p, (q - 1) * plane + out_off, am);
#pragma unroll
        for (int i = 0; i < 10; ++i) {
            A2[i] = PK<R>::mk(A2[i].y, ap[i]);
            ap[i] = R(0);
        }
    }
}

}  // namespace lbf
