// lbf_repulsive.cu -- REPULSIVE_FLUX (lb_cuda_repulsive_module.f90:19-292):
// a film-repulsion force between facing interfaces, computed before each step
// from the step's phi and read by the fused step's moments prologue
// (lb_cuda_moments_module.f90:148-160).  Two passes: the unit normals of the
// phi gradient (compute_norm's aux 1-3, lb_cuda_auxfields_module.f90:72-112),
// then per interfacial node the window scan for the facing partner and the
// pair's force (the reference's thinfilm_scan_mark_kernel and
// repulsive_flux_normal_kernel in one pass: the partner's offset is not kept).
// FP64, as the reference's (real(kind=db)).
#include <type_traits>

#include "lbf_chain.cuh"
#include "lbf_internal.h"
#include "lbf_stream.cuh"

namespace lbf {
namespace {

template <typename Fn> cudaError_t by_storage(int storage, Fn&& fn) {
    switch (storage) {
        case 0: return fn(float{});
        case 1: return fn(__half{});
        case 2: return fn(__nv_bfloat16{});
        case 3: return fn(double{});
    }
    return cudaErrorInvalidValue;
}

// index of (i, j, k) folded into the box on periodic axes; -1 beyond a
// non-periodic face (the reference's halo there: isfluid 1, phi 0, aux 0)
__device__ __forceinline__ long long wrap_idx(const RepulsiveArgs& a, int i, int j, int k) {
    bool ok = true;
    const int x = wrap_coord(i, a.nx, a.pbx, ok), y = wrap_coord(j, a.ny, a.pby, ok);
    const int z = wrap_coord(k, a.nz, a.pbz, ok);
    return ok ? ((long long)z * a.ny + y) * a.nx + x : -1;
}

// phi as the pair search reads it: after the mass correction of the step's
// input (thinfilm_scan_mark_cuda runs after bcs_mesoscopic_phifields,
// integrator_module.f90:297-328); the normals are compute_norm's, from the
// uncorrected phi
template <typename SP> struct SearchPhi {
    const SP* ph;
    double corr;
    bool mc;
    __device__ SearchPhi(const RepulsiveArgs& a) : ph(static_cast<const SP*>(a.phi)), corr(0.0) {
        mc = mass_corr(a.mass, corr);
    }
    __device__ double operator()(long long i) const {
        const double v = (double)ph[i];
        return mc ? mass_corrected<SP>(v, corr) : v;
    }
};
// q = phi (1 - phi) of phi clipped to [0, 1]
__device__ __forceinline__ double q_of(double phi) {
    const double c = fmin(fmax(phi, 0.0), 1.0);
    return c * (1.0 - c);
}
__device__ __forceinline__ bool is_fluid(const RepulsiveArgs& a, long long g) {
    if (!a.isf) return true;
    const int f = a.isf[g];
    return f == 1 || f == -1;
}

// A CTA works on a tile of RX x RY x RZ nodes.
constexpr int RX = 16, RY = 8, RZ = 8, RTILE = RX * RY * RZ, RTHREADS = 256;
constexpr int RH = 3;  // the search window
constexpr int RHX = RX + 2 * RH, RHY = RY + 2 * RH, RHZ = RZ + 2 * RH, RHALO = RHX * RHY * RHZ;

__device__ __forceinline__ void tile_origin(const RepulsiveArgs& a, int& X0, int& Y0, int& Z0) {
    const unsigned gx = (a.nx + RX - 1) / RX, gy = (a.ny + RY - 1) / RY;
    const unsigned b = blockIdx.x;
    X0 = (int)(b % gx) * RX;
    Y0 = (int)((b / gx) % gy) * RY;
    Z0 = (int)(b / (gx * gy)) * RZ;
}

// n = g / (|g| + 1e-9) (3 x N, FP64) on the fluid nodes with q >= q_th: the
// only ones that the search compares (a partner passes the same threshold as
// the node itself), so the others' slots keep whatever they hold.
template <typename SP> __global__ void __launch_bounds__(RTHREADS, 3) rep_normals_kernel(const RepulsiveArgs a) {
    chain_begin();
    const long long N = (long long)a.nx * a.ny * a.nz;
    const SearchPhi<SP> PH(a);
    int X0, Y0, Z0;
    tile_origin(a, X0, Y0, Z0);
    for (int t = threadIdx.x; t < RTILE; t += RTHREADS) {
        const int x = X0 + t % RX, y = Y0 + (t / RX) % RY, z = Z0 + t / (RX * RY);
        if (x >= a.nx || y >= a.ny || z >= a.nz) continue;
        const long long g = ((long long)z * a.ny + y) * a.nx + x;
        if (!is_fluid(a, g) || !(q_of(PH(g)) >= a.q_th)) continue;
        // the three coordinates of each axis, folded into the box once; -1
        // beyond a non-periodic face, where phi is 0
        int cx[3], cy[3], cz[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bool ok = true;
            cx[d] = wrap_coord(x + d - 1, a.nx, a.pbx, ok);
            if (!ok) cx[d] = -1;
            ok = true;
            cy[d] = wrap_coord(y + d - 1, a.ny, a.pby, ok);
            if (!ok) cy[d] = -1;
            ok = true;
            cz[d] = wrap_coord(z + d - 1, a.nz, a.pbz, ok);
            if (!ok) cz[d] = -1;
        }
        double gx, gy, gz;
        iso_grad<double>(
            [&](int p, int q, int r) {
                const int i = cx[p + 1], j = cy[q + 1], k = cz[r + 1];
                return (i | j | k) < 0 ? 0.0 : (double)PH.ph[((long long)k * a.ny + j) * a.nx + i];
            },
            gx, gy, gz);
        const double den = sqrt(gx * gx + gy * gy + gz * gz) + 1.0e-9;
        a.nrm[g] = gx / den; a.nrm[N + g] = gy / den; a.nrm[2 * N + g] = gz / den;
    }
}

// a vector of components within [-1, 1] in signed bytes (1 = 127)
__device__ __forceinline__ int pack_normal(float x, float y, float z) {
    const int a = __float2int_rn(127.f * x), b = __float2int_rn(127.f * y), c = __float2int_rn(127.f * z);
    return (a & 255) | (b & 255) << 8 | (c & 255) << 16;
}
// the most that the product of two packed unit vectors is off their FP64 one,
// in units of 1 / 127^2: sum of |127 a| / 2 + |127 b| / 2 + 1/4 over the
// components, at most 127 sqrt(3) + 3/4
constexpr int DOT_ONE = 127 * 127, DOT_ERR = 224;

// the force of each node (3 x N in the arithmetic type R; 0 where no pair).
// The search tests 342 neighbours of every interfacial node, in FP64 in the
// reference.  Here a CTA stages q (FP32) and the normal (bytes) of its tile
// and the 3-node halo in shared memory, collects its interfacial nodes, and
// each thread scans the window of one of them on the staged values, with
// margins wider than their rounding (q: 1e-6 against at most 3e-8; normals:
// DOT_ERR).  What passes, a few neighbours where interfaces face each other
// and none elsewhere, is decided on the FP64 values, so the partner is the one
// of the full search.  A tile whose normals all lie within a cone too narrow
// for a facing pair scans nothing.
// Bound by the issue of the scan (6 instructions a neighbour) and of the
// staging.  12 droplets in 112 x 96 x 88 (250 thousand interfacial nodes), both
// kernels: 1.52 ms for the FP64 scan of every neighbour from global memory,
// 0.35 ms with q staged and the normals tested one by one, 0.16 ms now.
template <typename SP, typename R> __global__ void __launch_bounds__(RTHREADS) rep_force_kernel(const RepulsiveArgs a) {
    __shared__ float2 sq[RHALO];  // q, packed normal
    __shared__ unsigned short list[RTILE];
    __shared__ int count, any_nan, narrow;
    __shared__ float sum[3];
    const long long N = (long long)a.nx * a.ny * a.nz;
    R* out = static_cast<R*>(a.force);
    const double eps = 1.0e-9;
    chain_begin();
    const SearchPhi<SP> PH(a);
    int X0, Y0, Z0;
    tile_origin(a, X0, Y0, Z0);
    if (threadIdx.x == 0) {
        count = any_nan = 0;
        narrow = DOT_ONE;
        sum[0] = sum[1] = sum[2] = 0.f;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < RTILE; t += RTHREADS) {
        const int x = X0 + t % RX, y = Y0 + (t / RX) % RY, z = Z0 + t / (RX * RY);
        if (x >= a.nx || y >= a.ny || z >= a.nz) continue;
        const long long g = ((long long)z * a.ny + y) * a.nx + x;
        // every node's force is 0 until a pair is found
        out[g] = R(0); out[N + g] = R(0); out[2 * N + g] = R(0);
        if (is_fluid(a, g) && q_of(PH(g)) >= a.q_th) list[atomicAdd(&count, 1)] = (unsigned short)t;
    }
    __syncthreads();
    const int n = count;
    if (n == 0) return;
    const float q_min = (float)a.q_th - 1.0e-6f;
    float m0 = 0.f, m1 = 0.f, m2 = 0.f;
    for (int i = threadIdx.x; i < RHALO; i += RTHREADS) {
        const long long g = wrap_idx(a, X0 + i % RHX - RH, Y0 + (i / RHX) % RHY - RH, Z0 + i / (RHX * RHY) - RH);
        float q = 0.f, n0 = 0.f, n1 = 0.f, n2 = 0.f;  // beyond a non-periodic face: phi 0, normal 0
        if (g >= 0) {
            if (!is_fluid(a, g)) {
                q = -1.f;
            } else {
                const double qd = q_of(PH(g));
                q = (float)qd;
                if (qd >= a.q_th) {
                    n0 = (float)a.nrm[g]; n1 = (float)a.nrm[N + g]; n2 = (float)a.nrm[2 * N + g];
                    if (isnan(n0 + n1 + n2)) any_nan = 1;
                }
            }
        }
        sq[i] = make_float2(q, __int_as_float(pack_normal(n0, n1, n2)));
        m0 += n0; m1 += n1; m2 += n2;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m0 += __shfl_xor_sync(0xffffffffu, m0, o);
        m1 += __shfl_xor_sync(0xffffffffu, m1, o);
        m2 += __shfl_xor_sync(0xffffffffu, m2, o);
    }
    if (threadIdx.x % 32 == 0) {
        atomicAdd(&sum[0], m0); atomicAdd(&sum[1], m1); atomicAdd(&sum[2], m2);
    }
    __syncthreads();
    // a comparison with NaN is false, so such a normal faces everything: no
    // test on the packed values then
    int dot_max = any_nan ? 4 * DOT_ONE : (int)floor(fmin(fmax(a.cos_opp_t, -2.0), 2.0) * DOT_ONE) + DOT_ERR;
    if (!any_nan) {
        // the cone around the mean normal: vectors of length <= 1 whose product
        // with the axis is at least d have products of at least 2 d^2 - 1
        const float len = sqrtf(sum[0] * sum[0] + sum[1] * sum[1] + sum[2] * sum[2]);
        const float inv = len > 0.f ? 1.f / len : 0.f;
        const int axis = pack_normal(sum[0] * inv, sum[1] * inv, sum[2] * inv);
        int least = DOT_ONE;
        for (int i = threadIdx.x; i < RHALO; i += RTHREADS) {
            const float2 v = sq[i];
            if (v.x >= q_min) least = min(least, __dp4a(__float_as_int(v.y), axis, 0));
        }
        least = __reduce_min_sync(0xffffffffu, least);
        if (threadIdx.x % 32 == 0) atomicMin(&narrow, least);
        __syncthreads();
        const float d = (float)(narrow - DOT_ERR) / DOT_ONE;
        if (d > 0.f && 2.f * d * d - 1.f > (float)a.cos_opp_t + 1.0e-3f) return;
    }
    for (int e = threadIdx.x; e < n; e += RTHREADS) {
        const int t = list[e];
        const int lx = t % RX, ly = (t / RX) % RY, lz = t / (RX * RY);
        const int x = X0 + lx, y = Y0 + ly, z = Z0 + lz;
        const long long g = ((long long)z * a.ny + y) * a.nx + x;
        const int c = ((lz + RH) * RHY + (ly + RH)) * RHX + (lx + RH);
        const double loc_phi = PH(g);
        const double qloc = q_of(loc_phi);
        const double nix = a.nrm[g], niy = a.nrm[N + g], niz = a.nrm[2 * N + g];
        const float qf = sq[c].x, q_tol = 0.1f * fmaxf(qf, 1.0e-12f) + 1.0e-6f;
        const float q_lo = fmaxf(q_min, qf - q_tol), q_hi = qf + q_tol;
        const int np = __float_as_int(sq[c].y);
        // scan and mark (lb_cuda_repulsive_module.f90:63-150): nearest facing
        // partner of similar q, ties to the larger facing factor; x outermost
        int best_r2 = 1 << 30;
        double best_face = -1.0;
        int bi = 0, bj = 0, bk = 0;
#pragma unroll 1
        for (int di = -RH; di <= RH; ++di) {
            // neighbours of this x offset that pass the staged tests: bit
            // 7 (dj + 3) + (dk + 3), the reference's order of the scan
            const float2* col = sq + c + di;
            unsigned m[2] = {0, 0};  // dj < 1, dj >= 1
#pragma unroll
            for (int dj = -RH; dj <= RH; ++dj)
#pragma unroll
                for (int dk = -RH; dk <= RH; ++dk) {
                    const float2 v = col[(dk * RHY + dj) * RHX];
                    const int bit = 7 * (dj + RH) + (dk + RH);
                    const bool pass = (v.x >= q_lo) & (v.x <= q_hi) & (__dp4a(__float_as_int(v.y), np, 0) <= dot_max);
                    m[bit >= 28] |= pass ? 1u << (bit >= 28 ? bit - 28 : bit) : 0u;
                }
            if (di == 0) m[0] &= ~(1u << 24);  // the node itself
            unsigned long long left = m[0] | ((unsigned long long)m[1] << 28);
            while (left) {
                const int bit = __ffsll(left) - 1;
                left &= left - 1;
                const int row = (bit * 37) / 256;  // bit / 7 of 0 .. 48
                const int dj = row - RH, dk = bit - 7 * row - RH;
                const int r2 = di * di + dj * dj + dk * dk;
                if (r2 > best_r2) continue;
                // the reference's tests, FP64
                const long long nb = wrap_idx(a, x + di, y + dj, z + dk);
                if (nb >= 0 && !is_fluid(a, nb)) continue;
                const double qn = nb < 0 ? 0.0 : q_of(PH(nb));
                if (qn < a.q_th || fabs(qn - qloc) > 0.1 * fmax(qloc, 1.0e-12)) continue;
                const double dotn = nb < 0 ? 0.0 : nix * a.nrm[nb] + niy * a.nrm[N + nb] + niz * a.nrm[2 * N + nb];
                if (dotn > a.cos_opp_t) continue;
                const double face = 0.5 * (1.0 - dotn);
                if (r2 < best_r2 || face > best_face) {
                    best_r2 = r2; best_face = face; bi = di; bj = dj; bk = dk;
                }
            }
        }
        // normal repulsive flux (lb_cuda_repulsive_module.f90:194-289)
        const double q1 = loc_phi * (1.0 - loc_phi);
        if (best_r2 < (1 << 30) && q1 > eps) {
            double dx = bi, dy = bj, dz = bk;
            const double r = sqrt(dx * dx + dy * dy + dz * dz);
            dx /= r; dy /= r; dz /= r;
            const long long nb = wrap_idx(a, x + bi, y + bj, z + bk);
            const double n2x = nb < 0 ? 0.0 : a.nrm[nb], n2y = nb < 0 ? 0.0 : a.nrm[N + nb];
            const double n2z = nb < 0 ? 0.0 : a.nrm[2 * N + nb];
            const double face = fmax(0.0, -(nix * n2x + niy * n2y + niz * n2z));
            if (face > eps) {
                double nsx = nix - n2x, nsy = niy - n2y, nsz = niz - n2z;
                const double nsm = sqrt(nsx * nsx + nsy * nsy + nsz * nsz);
                if (nsm <= eps) {
                    nsx = dx; nsy = dy; nsz = dz;
                } else {
                    nsx /= nsm; nsy /= nsm; nsz /= nsm;
                }
                if (dx * nsx + dy * nsy + dz * nsz < 0) { nsx = -nsx; nsy = -nsy; nsz = -nsz; }
                const double phi2 = nb < 0 ? 0.0 : PH(nb);
                const double qpair = 0.5 * (q1 + phi2 * (1.0 - phi2));
                const double qcl = fmin(fmax(qpair, eps), 0.25 - eps);
                const double arg = 1.0 / (2.0 * sqrt(qcl));
                if (arg > 1.0) {
                    const double wfilm = a.width * log(arg + sqrt(arg * arg - 1.0));
                    if (wfilm > 0) {
                        const double wd = 1.0 / (1.0 + pow(wfilm, 4.0));
                        const double s = a.a_rep * wd * qcl * face;
                        const double fx = s * nsx, fy = s * nsy, fz = s * nsz;
                        const double cap = 1.5 * (fabs(fx) + fabs(fy) + fabs(fz));
                        const double sc = fmin(1.0, loc_phi / fmax(cap, 1.0e-9));
                        out[g] = (R)(fx * sc); out[N + g] = (R)(fy * sc); out[2 * N + g] = (R)(fz * sc);
                    }
                }
            }
        }
    }
}

}  // namespace

cudaError_t launch_repulsive(int storage, const RepulsiveArgs& a, cudaStream_t st) {
    // one CTA per tile: at most (2^31 - 1) nodes, so the grid fits in 31 bits
    const long long tiles = (long long)((a.nx + RX - 1) / RX) * ((a.ny + RY - 1) / RY) * ((a.nz + RZ - 1) / RZ);
    return by_storage(storage, [&](auto tag) {
        using S = decltype(tag);
        using SP = typename PhiStore<S>::type;
        using R = typename std::conditional<sizeof(S) == 8, double, float>::type;
        const cudaError_t e = launch_chained(rep_normals_kernel<SP>, dim3((unsigned)tiles), RTHREADS, 0, st, a);
        if (e != cudaSuccess) return e;
        return launch_chained(rep_force_kernel<SP, R>, dim3((unsigned)tiles), RTHREADS, 0, st, a);
    });
}

}  // namespace lbf
