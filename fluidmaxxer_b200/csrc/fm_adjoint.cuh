// fm_adjoint.cuh -- reverse-mode (adjoint) kernels of the coupled step.
//
// Forward step s+1 maps the state X_s = (f_s, g_s, phi_s, q_s) to X_{s+1};
// phi_s is the AD scalar computed during step s (the LDF source of step s+1
// reads it).  f_s is held as the fused kernel holds it: at x = 0 the
// VelocityDirichletNEQ values the next pull reads, derived from f_s at x = 1.
// Given the adjoint lambda_{s+1} = dL/dX_{s+1}, one kernel produces lambda_s:
//
//   k_adj_step  per cell: gather lambda f_{s+1} and lambda g_{s+1} by the
//               transposed pull from the adjoints of the pulled populations
//               the backward step before left (each population was read by the
//               cells that pulled it: neighbour pull, keep-local, own-opposite
//               bounce-back, obstacle reversal), move the NEQ inlet's adjoint
//               from x = 0 into x = 1, recompute the forward step at the cell
//               (the same arithmetic as k_coupled_step), then apply in reverse
//               the AD boundaries, the D3Q7 collision, the LDF source, the
//               coupling velocity, the pressure outlet and the NS collision.
//               Writes the adjoints of the populations this step pulled (lfi,
//               lgi), lambda(phi_s), lambda(q_s) and accumulates the gradients
//               of the isotherm parameters and of the porosity field.
//
// The adjoint state therefore travels as (lfi, lgi): a gather at the start of
// the next step takes the place of a pass of its own over all 26 planes.
//
// Non-smooth points take the derivative of the branch the forward took (the
// phi clamp, max(c, eps), the porosity clamp).  Supported set-up: BGK or
// porous collision, NEQ inlet on the full x = 0 plane (or none), pressure
// outlet on the full x = nx-1 plane (or none), AD Dirichlet / Neumann on the
// full planes (or none), linear or Langmuir isotherm, the outlet probe on the
// x = nx-1 plane, even nx.
#pragma once

#include "fm_kernels.cuh"

namespace fm {

// Ordinary coherent loads that stay behind pdl_wait (as ld_pop); with a condition,
// predicated, and 0 where it is false.
__device__ __forceinline__ float ld_adj(const float* p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_adj(const double* p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_adj(const float* p, bool on)
{
    float v;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f32 %0, 0f00000000; @q ld.global.f32 %0, [%1]; }"
                 : "=&f"(v) : "l"(p), "r"((uint32_t)on));
    return v;
}
__device__ __forceinline__ double ld_adj(const double* p, bool on)
{
    double v;
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; mov.f64 %0, 0d0000000000000000; @q ld.global.f64 %0, [%1]; }"
                 : "=&d"(v) : "l"(p), "r"((uint32_t)on));
    return v;
}

template <typename T, typename QT>
struct AdjArgs {
    using R = typename Pop<T>::R;
    StepArgs<T, QT> a;              // forward step from X_s (fA = f_s, gA = g_s, phi = phi_s, q = q_s)
    // The launches before a backward step write all of these, and it may start
    // while they drain: inputs are read by ld_adj behind pdl_wait, and nothing is
    // declared __restrict__, which would let a load take the read-only path or
    // move above the wait.
    const R* lfi1;                  // adjoints of the D3Q19 populations step s+2 pulled [19][ns]
    const R* lgi1;                  // the same of the D3Q7 populations [7][ns]
    const R* lphi1;                 // lambda phi_{s+1}
    const R* lq1;                   // lambda q_{s+1}
    R* lfi;                         // out: adjoints of the D3Q19 populations step s+1 pulls
    R* lgi;                         // out: the same of the D3Q7 populations
    R* lphi0;                       // out: lambda phi_s
    R* lq0;                         // out: lambda q_s
    R* x1;                          // [19][rows]: f_{s+1} at x = 1 in, f_s at x = 1 out
    double* gpor;                   // += dL/d porosity per cell (porous collision)
    double* gpar;                   // += dL/d (isotherm a, b, k), per warp [warps][3]
    R wl;                           // loss weight on phi_{s+1} of the outlet plane (0: not sampled)
    int first;                      // no backward step before: lfi1, lgi1 are zero
};

// c v for a velocity component c of direction K (v, 0 or -v)
template <int C, typename R>
__device__ __forceinline__ R times_c(R v)
{
    return C == 0 ? R(0) : (C > 0 ? v : -v);
}

// d feq_K / du of the second-order equilibrium: w rho (3 c + 9 (c.u) c - 3 u)
template <int K, typename R>
__device__ __forceinline__ void dfeq_du(R rho, R ux, R uy, R uz, R& gx, R& gy, R& gz)
{
    const R e9 = R(9) * cdot<cx19(K), cy19(K), cz19(K)>(ux, uy, uz);
    const R wr = w19<R>(K) * rho;
    gx = wr * ((R(3 * cx19(K)) + times_c<cx19(K)>(e9)) - R(3) * ux);
    gy = wr * ((R(3 * cy19(K)) + times_c<cy19(K)>(e9)) - R(3) * uy);
    gz = wr * ((R(3 * cz19(K)) + times_c<cz19(K)>(e9)) - R(3) * uz);
}

// feq_K / (w_K rho), m = 1.5 u^2
template <int K, typename R>
__device__ __forceinline__ R poly19(R ux, R uy, R uz, R m)
{
    const R e = cdot<cx19(K), cy19(K), cz19(K)>(ux, uy, uz);
    return R(1) + R(3) * e + R(4.5) * e * e - m;
}

// f(std::integral_constant<int, K>) for K = 0..18
template <typename F, int... Ks>
__device__ __forceinline__ void each19(F f, std::integer_sequence<int, Ks...>)
{
    (f(std::integral_constant<int, Ks>{}), ...);
}

template <typename R>
__device__ __forceinline__ R warp_sum_r(R v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The transposed pull of direction J at a cell away from the y/z faces: the
// sum of the adjoints of the pulls that read the cell's population J -- by the
// cell at c + c_J, by the cell itself where that lies outside (keep-local), by
// its own opposite direction (a link to an obstacle at c + c_J, or an obstacle
// cell, whose bits lk 1..18 are all set).
template <int J, bool BB, typename R>
__device__ __forceinline__ R gather19_fast(const R* base, uint32_t ns, int nx, int nxy, int px, bool xlo,
                                           bool xhi, uint32_t lk, bool solid)
{
    constexpr int CX = cx19(J), CY = cy19(J), CZ = cz19(J), O = opp19(J);
    if (J == 0) return ld_adj(base);
    const bool own = BB && ((lk >> O) & 1u);
    const bool out = CX != 0 && (CX > 0 ? xhi : xlo);    // c + c_J beyond an x-face
    const bool keep = CX != 0 && (CX > 0 ? xlo : xhi);   // c - c_J beyond an x-face: the cell kept its own value
    uint32_t off = (uint32_t)J * ns + (uint32_t)(CX + CY * nx + CZ * nxy);
    if (out) off -= (uint32_t)(CX * nx);                 // periodic x
    if (own) off = (uint32_t)O * ns;
    R v = ld_adj(base + off);                            // in the array in any case
    if (out && !px && !own) v = R(0);
    if (CX != 0) {
        const bool too = keep && !px && !solid;
        const R k = ld_adj(base + (uint32_t)J * ns, too);
        if (too) v += k;
    }
    return v;
}
// the same for any cell
template <int J, bool BB, typename R>
__device__ __forceinline__ R gather19(const R* l, uint32_t ns, uint32_t c, const Nbr& nb, uint32_t w,
                                      bool solid)
{
    constexpr int CX = cx19(J), CY = cy19(J), CZ = cz19(J), O = opp19(J);
    if (J == 0) return ld_adj(l + c);
    const bool in_o = nb.inside<-CX, -CY, -CZ>(), in_j = nb.inside<CX, CY, CZ>();
    const bool link = BB && ((w >> O) & 1u);
    R v = R(0);
    if (in_o && !link && !solid) v += ld_adj(l + ((uint32_t)J * ns + (uint32_t)nb.src<-CX, -CY, -CZ>()));
    if (!in_j && !solid) v += ld_adj(l + ((uint32_t)J * ns + c));
    if (solid || (in_o && link)) v += ld_adj(l + ((uint32_t)O * ns + c));
    return v;
}
// D3Q7 has no reflection
template <int J, typename R>
__device__ __forceinline__ R gather7_fast(const R* base, uint32_t ns, int nx, int nxy, int px, bool xlo,
                                          bool xhi)
{
    return gather19_fast<J, false>(base, ns, nx, nxy, px, xlo, xhi, 0u, false);
}
static_assert(cx19(1) == cx7(1) && cx19(2) == cx7(2) && cy19(3) == cy7(3) && cy19(4) == cy7(4) && cz19(5) == cz7(5) &&
                  cz19(6) == cz7(6),
              "the D3Q7 directions are the first seven of D3Q19");

// threads per block, and resident blocks per SM k_adj_step is compiled for: 80
// registers (FP32) and 168 (FP64), the recomputed forward and the adjoint both
// live.  A gradient of 240 steps at 48x80x80: FP32 6 blocks 19.6 ms, 7 19.8, 8
// 19.7; FP64 2 blocks 36.4 ms, 3 32.5, 4 31.3 (but 24x40x40 8.1, 7.6, 8.1).
constexpr int kAdjThreads = 128;
template <typename T>
constexpr int kAdjBlocks = sizeof(T) == 8 ? 3 : 6;

// Bound by latency and instruction issue (24 FP32 warps an SM, 2520 instructions
// each, 48% of cycles issuing).  It replaces a cell kernel, a stream kernel and an inlet kernel, which
// passed the 26 adjoint planes through memory once more (564 against 352 B a
// cell), formed every product with the zero velocity components and took the
// neighbour table in every warp.  All loads of populations and adjoints come
// first, so a cell waits for memory once: a gradient of 240 steps at 48x80x80
// took 26.7 ms with the three kernels, 21.5 with one that loads where it uses,
// 19.6 with this order (FP64 49.7, 43.8, 32.5).
template <typename T, typename QT, bool POROUS>
__global__ void __launch_bounds__(kAdjThreads, kAdjBlocks<T>) k_adj_step(const AdjArgs<T, QT> A)
{
    using R = typename Pop<T>::R;
    const StepArgs<T, QT>& a = A.a;
    __shared__ R line[kAdjThreads / 32][20];   // one inlet row at a time, per warp
    const uint32_t cg = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = cg < (uint32_t)a.n;
    const uint32_t c = active ? cg : (uint32_t)a.n - 1u;
    const int lane = threadIdx.x & 31;
    const uint32_t w = __ldg(a.cellw + c);
    pdl_wait();
    const bool solid = !POROUS && (w & kSolid);
    const bool xlo = (w & kXLo) != 0u, xhi = (w & kXHi) != 0u;
    const uint32_t ns = a.ns;
    const int nxy = a.nx * a.ny;
    const uint32_t lk = solid ? 0x7fffeu : w;
    const bool face = __any_sync(0xffffffffu, w & kFaceYZ);
    int x = 1, y = 1, z = 1;
    if (face) cell_xyz(c, a.nx, a.ny, a.div_nx, a.div_nxy, x, y, z);
    const Nbr nb(x, y, z, a.nx, a.ny, a.nz, a.px, a.py, a.pz);

    // ---- forward recompute of the NS part ----
    R fi[19];
    if (face) pull19_all<T, !POROUS>(fi, a.fA, ns, c, nb, w, a.f_shift, Seq19{});
    else pull19_fast_all<T, !POROUS>(fi, a.fA + c, ns, a.nx, nxy, a.px, xlo, xhi, lk, R(0), Seq19{});
    R gi[7];
    if (face) pull7(a, c, nb, gi);
    else pull7_fast_all<T>(gi, a.gA + c, ns, a.nx, nxy, a.px, xlo, xhi, a.g_shift, Seq7{});
    R lg[7];
    if (face) {
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            if constexpr (K < 7) lg[K] = gather19<K, false>(A.lgi1, ns, c, nb, 0u, false);
        }, Seq19{});
    } else {
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            if constexpr (K < 7) lg[K] = gather7_fast<K>(A.lgi1 + c, ns, a.nx, nxy, a.px, xlo, xhi);
        }, Seq19{});
    }
    R lf[19];
    if (face)
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            lf[K] = gather19<K, !POROUS>(A.lfi1, ns, c, nb, w, solid);
        }, Seq19{});
    else
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            lf[K] = gather19_fast<K, !POROUS>(A.lfi1 + c, ns, a.nx, nxy, a.px, xlo, xhi, lk, solid);
        }, Seq19{});
    R rho = R(0), ubx = R(0), uby = R(0), ubz = R(0), ux = R(0), uy = R(0), uz = R(0), por = R(1);
    bool por_free = false;   // porosity strictly inside [0,1]: the clamp passes the derivative
    if (!solid) {
        R jx, jy, jz;
        moments19(fi, rho, jx, jy, jz, Seq19{});
        if (!(rho > R(0))) { rho = a.rho0; jx = jy = jz = R(0); }
        const R inv = R(1) / rho;
        ubx = jx * inv; uby = jy * inv; ubz = jz * inv;
        ux = ubx; uy = uby; uz = ubz;
        if (POROUS) {
            R ph = __ldg(a.porosity + c);
            por_free = ph > R(0) && ph < R(1);
            if (ph < R(0)) ph = R(0);
            if (ph > R(1)) ph = R(1);
            por = ph;
            ux *= ph; uy *= ph; uz *= ph;
        }
    }
    const R m15 = R(1.5) * (ux * ux + uy * uy + uz * uz);
    // post-collision populations (BGK: fi + omega (feq - fi); obstacle: fi), in place
    if (!solid)
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            const R feq = w19<R>(K) * rho * poly19<K>(ux, uy, uz, m15);
            fi[K] = fi[K] + a.omega * (feq - fi[K]);
        }, Seq19{});
    // their moments (the x-1 neighbour's velocity for the outlet)
    R rh, hx, hy, hz;
    moments19(fi, rh, hx, hy, hz, Seq19{});
    const R ih = (rh > R(0)) ? (R(1) / rh) : R(0);
    const R uhx = hx * ih, uhy = hy * ih, uhz = hz * ih;
    // the coupling velocity of the populations after the outlet boundary
    const bool outlet = a.fuse_outlet && xhi;
    R rp = rh, ip = ih, uax = uhx, uay = uhy, uaz = uhz;
    R uNx = R(0), uNy = R(0), uNz = R(0);
    if (__any_sync(0xffffffffu, outlet)) {
        uNx = __shfl_up_sync(0xffffffffu, uhx, 1);
        uNy = __shfl_up_sync(0xffffffffu, uhy, 1);
        uNz = __shfl_up_sync(0xffffffffu, uhz, 1);
        if (outlet) {
            R fp[19], jx, jy, jz;
            const R mN = R(1.5) * (uNx * uNx + uNy * uNy + uNz * uNz);
            each19([&](auto k) {
                constexpr int K = decltype(k)::value;
                fp[K] = w19<R>(K) * a.rho_out * poly19<K>(uNx, uNy, uNz, mN);
            }, Seq19{});
            moments19(fp, rp, jx, jy, jz, Seq19{});
            ip = (rp > R(0)) ? (R(1) / rp) : R(0);
            uax = jx * ip; uay = jy * ip; uaz = jz * ip;
        }
    }
    if (!a.coupling) uax = uay = uaz = R(0);

    // ---- forward recompute of the AD part ----
    R gs = gi[0];
#pragma unroll
    for (int k = 1; k < 7; ++k) gs += gi[k];
    const bool phi_free = !(gs < a.min_conc);
    const R phi = phi_free ? gs : a.min_conc;
    const R om = a.tau_ad ? R(1) / __ldg(a.tau_ad + c) : a.omega_ad;
    const bool region = a.isotherm != 0 && (w & kRegion);

    // ---- adjoint of the AD boundaries and collision ----
    if (__any_sync(0xffffffffu, xlo || xhi)) {
        if (a.fuse_dirichlet && xlo) {
#pragma unroll
            for (int k = 0; k < 7; ++k) lg[k] = R(0);
        }
        if (a.fuse_neumann) {
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const R right = __shfl_down_sync(0xffffffffu, lg[k], 1);
                if (xhi) lg[k] = R(0);
                else if (w & kXHi1) lg[k] += right;
            }
        }
    }
    R lphi = ld_adj(A.lphi1 + c) + (xhi ? A.wl : R(0));
    R lS = R(0), lux = R(0), luy = R(0), luz = R(0);
    R bsum = lphi;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        R eu;
        if (k == 0) eu = R(0);
        else if (k == 1) eu = uax;
        else if (k == 2) eu = -uax;
        else if (k == 3) eu = uay;
        else if (k == 4) eu = -uay;
        else if (k == 5) eu = uaz;
        else eu = -uaz;
        bsum += lg[k] * om * w7<R>(k) * (R(1) + R(4) * eu);
        lS += lg[k] * w7<R>(k);
        const R t = lg[k] * om * w7<R>(k) * phi * R(4);
        if (k == 1) lux += t;
        else if (k == 2) lux -= t;
        else if (k == 3) luy += t;
        else if (k == 4) luy -= t;
        else if (k == 5) luz += t;
        else if (k == 6) luz -= t;
    }
    if (active) {
#pragma unroll
        for (int k = 0; k < 7; ++k)
            A.lgi[(uint32_t)k * ns + c] = (R(1) - om) * lg[k] + (phi_free ? bsum : R(0));
    }

    // ---- adjoint of the LDF source ----
    R lq = ld_adj(A.lq1 + c);
    R lphi0 = R(0);
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    if (region) {
        const R p0 = ld_adj(a.phi + c);
        const bool cfree = !(p0 < a.min_conc);
        const R ce = (cfree ? p0 : a.min_conc) - a.min_conc;
        const R qi = (R)ld_adj(a.q + c);
        R qeq, dqeq_dce, g_a, g_b;
        if (a.isotherm == 1) {
            qeq = a.iso_a * ce;
            dqeq_dce = a.iso_a;
            g_a = ce;
            g_b = R(0);
        } else {
            const R bc = a.iso_b * ce;
            const R den = R(1) + bc;
            qeq = a.iso_a * (bc / den);
            dqeq_dce = a.iso_a * a.iso_b / (den * den);
            g_a = bc / den;
            g_b = a.iso_a * ce / (den * den);
        }
        const R ldq = lq - lS;              // q' = q + dq, S = -dq
        const R lqeq = a.iso_k * ldq;
        g0 = (double)(lqeq * g_a);
        g1 = (double)(lqeq * g_b);
        g2 = (double)(ldq * (qeq - qi));
        lq = lq - a.iso_k * ldq;
        lphi0 = cfree ? lqeq * dqeq_dce : R(0);
    }
    if (active) {
        A.lphi0[c] = lphi0;
        A.lq0[c] = lq;
    }

    // ---- adjoint of the NS part ----
    pdl_launch_dependents();
    // The NEQ inlet in the fused representation: the stored x = 0 populations of
    // X_{s+1} are NEQ(f_{s+1} at x = 1) (src/boundary/ns/VelocityDirichletNEQ.cu:49-96),
    // f_B = feq(rho_N, u_BC) + f_N - feq(rho_N, u_N).  Per row, lane k (direction
    // k) moves the x = 0 adjoint into the x = 1 cell through the transposed
    // Jacobian (identity, the rho_N derivative of the two equilibria, the u_N
    // derivative of feq(rho_N, u_N)); the x = 0 adjoint is cleared.  nx is even,
    // so both cells are lanes of this warp.
    if (a.fuse_inlet) {
        R* const ln = line[threadIdx.x >> 5];
        const bool on = lane < 19;
        const int k = on ? lane : 0;
        const R cx = (R)((int)((kPX >> k) & 1u) - (int)((kMX >> k) & 1u));
        const R cy = (R)((int)((kPY >> k) & 1u) - (int)((kMY >> k) & 1u));
        const R cz = (R)((int)((kPZ >> k) & 1u) - (int)((kMZ >> k) & 1u));
        const R wk = k == 0 ? R(1) / R(3) : (k < 7 ? R(1) / R(18) : R(1) / R(36));
        for (uint32_t m = __ballot_sync(0xffffffffu, active && (w & kXLo1)); m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            const uint32_t c1 = cg - (uint32_t)lane + (uint32_t)src;   // the x = 1 cell
            R* const side = A.x1 + ((uint32_t)k * a.rows_stride + fastdiv(c1, a.div_nx));
            const R fN = ld_adj(side, on);
            if (on) *side = Pop<T>::ld(a.fA + (uint32_t)k * ns + c1, fshift<T>(k, a.f_shift));
            if (A.first) continue;
            if (lane == src - 1) {
#pragma unroll
                for (int j = 0; j < 19; ++j) ln[j] = lf[j];
            }
            __syncwarp();
            const R lB = on ? ln[k] : R(0);
            const R r = warp_sum_r(fN);
            const R jx = warp_sum_r(cx * fN), jy = warp_sum_r(cy * fN), jz = warp_sum_r(cz * fN);
            const R inv = (r > R(0)) ? (R(1) / r) : R(0);
            const R unx = jx * inv, uny = jy * inv, unz = jz * inv;
            const R cuB = R(3) * (cx * a.uin_x + cy * a.uin_y + cz * a.uin_z);
            const R cuN = R(3) * (cx * unx + cy * uny + cz * unz);
            const R pB = R(1) + cuB + R(0.5) * cuB * cuB -
                         R(1.5) * (a.uin_x * a.uin_x + a.uin_y * a.uin_y + a.uin_z * a.uin_z);
            const R pN = R(1) + cuN + R(0.5) * cuN * cuN - R(1.5) * (unx * unx + uny * uny + unz * unz);
            // d feq_k(r, u_N) / d u_N = w r (3 c + 9 (c.u) c - 3 u)
            const R e = cx * unx + cy * uny + cz * unz;
            const R gx = wk * r * (R(3) * cx + R(9) * e * cx - R(3) * unx);
            const R gy = wk * r * (R(3) * cy + R(9) * e * cy - R(3) * uny);
            const R gz = wk * r * (R(3) * cz + R(9) * e * cz - R(3) * unz);
            const R s1 = warp_sum_r(lB * wk * (pB - pN));
            const R Vx = warp_sum_r(lB * gx), Vy = warp_sum_r(lB * gy), Vz = warp_sum_r(lB * gz);
            if (on) ln[k] = lB + s1 - ((cx - unx) * Vx + (cy - uny) * Vy + (cz - unz) * Vz) * inv;
            __syncwarp();
            if (lane == src) {
#pragma unroll
                for (int j = 0; j < 19; ++j) lf[j] += ln[j];
            }
            if (lane == src - 1) {
#pragma unroll
                for (int j = 0; j < 19; ++j) lf[j] = R(0);
            }
            __syncwarp();
        }
    }
    if (a.coupling && rp > R(0)) {
        // u_adv = j(fp) / rho(fp)
#pragma unroll
        for (int k = 0; k < 19; ++k)
            lf[k] += (((R)cx19(k) - uax) * lux + ((R)cy19(k) - uay) * luy + ((R)cz19(k) - uaz) * luz) * ip;
    }
    // pressure outlet: fp(nx-1) = feq_out(rho_out, u of fh(nx-2))
    if (__any_sync(0xffffffffu, outlet)) {
        R lNx = R(0), lNy = R(0), lNz = R(0);
        if (outlet)
            each19([&](auto k) {
                constexpr int K = decltype(k)::value;
                R gx, gy, gz;
                dfeq_du<K>(a.rho_out, uNx, uNy, uNz, gx, gy, gz);
                lNx += lf[K] * gx; lNy += lf[K] * gy; lNz += lf[K] * gz;
                lf[K] = R(0);
            }, Seq19{});
        const R rx = __shfl_down_sync(0xffffffffu, lNx, 1);
        const R ry = __shfl_down_sync(0xffffffffu, lNy, 1);
        const R rz = __shfl_down_sync(0xffffffffu, lNz, 1);
        if ((w & kXHi1) && rh > R(0)) {
#pragma unroll
            for (int k = 0; k < 19; ++k)
                lf[k] += (((R)cx19(k) - uhx) * rx + ((R)cy19(k) - uhy) * ry + ((R)cz19(k) - uhz) * rz) * ih;
        }
    }
    // collision: fh = fi + omega (feq(rho, u) - fi), u = por * j / rho
    if (!solid) {
        R As = R(0), Vx = R(0), Vy = R(0), Vz = R(0);
        each19([&](auto k) {
            constexpr int K = decltype(k)::value;
            As += lf[K] * w19<R>(K) * poly19<K>(ux, uy, uz, m15);
            R gx, gy, gz;
            dfeq_du<K>(rho, ux, uy, uz, gx, gy, gz);
            Vx += lf[K] * gx; Vy += lf[K] * gy; Vz += lf[K] * gz;
        }, Seq19{});
        const R sc = a.omega * por / rho;
#pragma unroll
        for (int k = 0; k < 19; ++k)
            lf[k] = (R(1) - a.omega) * lf[k] + a.omega * As +
                    sc * (((R)cx19(k) - ubx) * Vx + ((R)cy19(k) - uby) * Vy + ((R)cz19(k) - ubz) * Vz);
        if (POROUS && active && por_free)
            A.gpor[c] += (double)(a.omega * (Vx * ubx + Vy * uby + Vz * ubz));
    }
    if (active) {
#pragma unroll
        for (int k = 0; k < 19; ++k) A.lfi[(uint32_t)k * ns + c] = lf[k];
    }
    // this warp's share of the isotherm gradients, in a place of its own (summed by
    // k_adj_fold at the end): no barrier and no atomics to three shared addresses
    if (__any_sync(0xffffffffu, region && active)) {
        const double s0 = warp_sum(active ? g0 : 0.0), s1 = warp_sum(active ? g1 : 0.0), s2 = warp_sum(active ? g2 : 0.0);
        if (lane == 0) {
            double* const p = A.gpar + (size_t)3 * (cg >> 5);
            p[0] += s0; p[1] += s1; p[2] += s2;
        }
    }
}

// the warps' shares of the isotherm gradients summed, in a fixed order
__global__ void __launch_bounds__(1024) k_adj_fold(const double* __restrict__ part, int nwarps, double* __restrict__ out)
{
    __shared__ double sh[32][3];
    double v[3] = {0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < nwarps; i += blockDim.x)
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] += part[(size_t)3 * i + j];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        v[j] = warp_sum(v[j]);
        if (lane == 0) sh[wid][j] = v[j];
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double s = warp_sum(lane < nw ? sh[lane][j] : 0.0);
            if (lane == 0) out[j] = s;
        }
    }
}

}  // namespace fm
