// Trajectory loss and its parameter gradient on the physics path (adjoint
// of the unrolled velocity-Verlet steps; the algebra is in adjoint.cuh).
//
// Passes over the state of step n (8 lanes per particle over the Verlet list,
// as the forward pair kernel):
//   k_loss_pairs   LJ energy and the RDF-bin occupancies h_b(x_n)
//   k_adj_bonded   per bonded term: its forces as dual numbers along w, so the
//                  tangent is the term's Hessian-vector product; loss gradient
//                  and the bonded-scale derivatives
//   k_adj_pair     per particle: sum over pairs of J_ij (w_i - w_j) with
//                  J = f I + 2 f' d d^T (f(r^2) the switched LJ force / r),
//                  the loss gradient (energy and RDF terms), sigma / epsilon
//                  derivatives chained through Lorentz-Berthelot; updates dL/dx
// Every per-lane sum is FP32; the energies, occupancies and parameter
// derivatives are reduced per block in FP64.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "adjoint.cuh"
#include "physkern.cuh"
#include "physmath.cuh"
#include "refdev.cuh"

namespace lima {
namespace {

constexpr int kAdjTB = 256;   // 32 particles x kGroup lanes
// Inside a checkpoint segment the pair list is rebuilt in place (particle
// order kept) every kListEpoch steps; the backward pass rebuilds the list of
// each epoch from its first state, which reproduces the forward's lists.
constexpr int kListEpoch = 10;

__device__ __forceinline__ float mimg_a(float d, float L, float invL) { return d - L * rintf(d * invL); }

// f(slot j, position) for one lane's entries of particle i's list, of the LANES
// lanes that share it: lane 8 h + g takes column g of the chunks h, h + LANES /
// 8, ... (nl_word), four entries per vector load and four gathers in flight.
template <int LANES, typename ID, typename F>
__device__ __forceinline__ void for_entries(const PhysDev& d, const float4* __restrict__ pos, int i, int lane, int cnt,
                                            F f) {
    using V = typename std::conditional<sizeof(ID) == 2, uint2, uint4>::type;
    constexpr int H = LANES / kGroup;
    const int g = lane % kGroup, h = lane / kGroup;
    const size_t cstride = (size_t)d.n_pad * kGroup;
    const V* __restrict__ col = reinterpret_cast<const V*>(d.nl) + (size_t)i * kGroup + g + h * cstride;
    for (int k = h * kListChunk + g; k < cnt; k += H * kListChunk, col += H * cstride) {
        const V v = __ldg(col);
        uint32_t j[4];
        if constexpr (sizeof(ID) == 2) {
            j[0] = v.x & 0xffffu;
            j[1] = v.x >> 16;
            j[2] = v.y & 0xffffu;
            j[3] = v.y >> 16;
        } else {
            j[0] = v.x;
            j[1] = v.y;
            j[2] = v.z;
            j[3] = v.w;
        }
        const int m = min(4, (cnt - k + kGroup - 1) / kGroup);   // words past the count are not ids
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; u++) p[u] = __ldg(pos + (u < m ? j[u] : j[0]));
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (u < m) f(j[u], p[u]);
    }
}

__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Quadratic B-spline bins of a distance: bins k0, k0+1, k0+2 with weights w
// and d w / d r (bin b is centred at (b + 1/2) dr).
__device__ __forceinline__ void bspline3(float r, float inv_dr, int& k0, float w[3], float dw[3]) {
    const float u = r * inv_dr - 0.5f;
    const float kc = rintf(u);
    const float t = u - kc;
    k0 = (int)kc - 1;
    w[0] = 0.5f * (0.5f - t) * (0.5f - t);
    w[1] = 0.75f - t * t;
    w[2] = 0.5f * (0.5f + t) * (0.5f + t);
    dw[0] = -(0.5f - t) * inv_dr;
    dw[1] = -2.f * t * inv_dr;
    dw[2] = (0.5f + t) * inv_dr;
}

// Switched LJ with 4 eps factored out: phi = 4 eps * ph, F_i = 4 eps * f * (x_i - x_j).
// Returns ph, f, df/d(r^2) and their sigma derivatives.
struct LJ1 {
    float ph, f, fp, dph_ds, df_ds;
};
// isig = 1 / sigma.
__device__ __forceinline__ LJ1 lj1(const PhysDev& d, float r2, float sig2, float isig) {
    const float u = rcp_newton(r2);
    const float s2 = sig2 * u, s6 = s2 * s2 * s2, s12 = s6 * s6;
    const float ph = s12 - s6;
    const float f = 6.f * u * (2.f * s12 - s6);
    const float fp = -6.f * u * u * (14.f * s12 - 4.f * s6);
    const float dph_ds = (12.f * s12 - 6.f * s6) * isig;
    const float df_ds = 6.f * u * (24.f * s12 - 6.f * s6) * isig;
    // C2 switch S(t), t = (rc^2 - r^2) / (rc^2 - r_on^2)
    const float t = __saturatef((d.rc2 - r2) * d.inv_sw_d);
    const float omt = 1.f - t;
    const float S = t * t * t * fmaf(t, fmaf(6.f, t, -15.f), 10.f);
    const float Sp = -30.f * t * t * omt * omt * d.inv_sw_d;
    const float Spp = 60.f * t * omt * (1.f - 2.f * t) * d.inv_sw_d * d.inv_sw_d;
    LJ1 o;
    o.ph = ph * S;
    o.f = f * S - 2.f * ph * Sp;
    o.fp = fp * S + 2.f * f * Sp - 2.f * ph * Spp;
    o.dph_ds = dph_ds * S;
    o.df_ds = df_ds * S - 2.f * dph_ds * Sp;
    return o;
}

struct AdjArgs {
    float dt;
    float le;          // w_energy / (N T) where this state carries a loss term, else 0
    float lr;          // 2 w_rdf / (N T) likewise
    float inv_dr;
    float supp2;       // (r_max + dr)^2
    int n_bins;
    int n_types;
    float4* lam_x;
    const float4* wv;
    float4* adj_term;
    const float* par;  // sigma[n_types], epsilon[n_types], scales
    double* gtheta;
    double2* gterm;    // per bonded term: dL/dc, dL/dk (c = r0 | theta0 | phi0)
};

// --------------------------------------------------------------- loss pass --
// A lane keeps occupancies of its own, one column of a [bins + 4][32] array per
// warp in shared memory (a row past either end takes the weights that fall
// outside, so no bin is tested): each of a pair's three weights is a plain load,
// add and store with no bank conflict and no atomic.  The sums are exact and so
// independent of their order: half weights (each pair is seen from both ends) as
// integers in units of 2^-32, in 32-bit columns, the additions that pass 2^32
// counted per bin by a shared atomic; the block's lanes are summed in FP64.
// 200 steps of 8,192 particles, 50 bins, on one B200: three 64-bit shared-memory
// atomics a pair 23.4 ms; this 10.7; FP32 columns, which round, 9.9; FP64 columns,
// twice the memory, 12.9 (32,024 particles, 128 bins, one lima_rdf: 176 us, 162,
// 300).
constexpr int kLossTB = 128;
// its static shared memory (warp energies and the LJ table), which counts
// towards the 48 KB that a launch gets without asking
constexpr size_t kLossStaticSmem = sizeof(double) * (kLossTB / 32) + sizeof(float2) * kMaxTypes * kMaxTypes;
constexpr size_t loss_smem(int n_bins) { return sizeof(uint32_t) * (n_bins + 4) * (32 * (kLossTB / 32) + 1); }
constexpr double kHistUnit = 1.0 / 4294967296.0;   // 2^-32
template <typename ID>
__global__ void __launch_bounds__(kLossTB) k_loss_pairs(PhysDev d, const float4* __restrict__ pos, int n_bins,
                                                        float inv_dr, float supp2, double inv_n,
                                                        double* __restrict__ U_out, double* __restrict__ h_out) {
    extern __shared__ uint32_t s_hist[];   // [warps][n_bins + 4][32], then the carries [n_bins + 4]
    __shared__ double s_e[kLossTB / 32];
    __shared__ float2 s_tab[kMaxTypes * kMaxTypes];
    const int nt2 = d.n_types * d.n_types, rows = n_bins + 4;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int q = threadIdx.x; q < nt2; q += blockDim.x) s_tab[q] = d.lj_table[q];
    uint32_t* mine = s_hist + (size_t)w * rows * 32 + lane;   // the lane's column
    uint32_t* carry = s_hist + (size_t)(kLossTB / 32) * rows * 32;
    for (int b = 0; b < rows; b++) mine[b * 32] = 0u;
    for (int b = threadIdx.x; b < rows; b += blockDim.x) carry[b] = 0u;
    __syncthreads();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kGroup;
    const int g = threadIdx.x % kGroup;
    float e = 0.f;
    if (i < d.n) {
        const float4 pi = pos[i];
        const float2* row = s_tab + __float_as_int(pi.w) * d.n_types;
        const int cnt = (int)d.nl_cnt[i];
        for_entries<kGroup, ID>(d, pos, i, g, cnt, [&](uint32_t, float4 pj) {
            const float dx = mimg_add(pi.x - pj.x, d.L, d.invL), dy = mimg_add(pi.y - pj.y, d.L, d.invL),
                        dz = mimg_add(pi.z - pj.z, d.L, d.invL);
            const float r2 = dx * dx + dy * dy + dz * dz;
            const float2 tab = row[__float_as_int(pj.w)];
            const float s2 = tab.x * rcp_newton(r2), s6 = s2 * s2 * s2;
            const float t = __saturatef((d.rc2 - r2) * d.inv_sw_d);   // 0 beyond r_c
            e += tab.y * fmaf(s6, s6, -s6) * (t * t * t * fmaf(t, fmaf(6.f, t, -15.f), 10.f));
            if (r2 < supp2) {
                int k0;
                float wt[3], dw[3];
                bspline3(sqrtf(r2), inv_dr, k0, wt, dw);
                uint32_t* q = mine + (k0 + 1) * 32;   // k0 is -1 .. n_bins
                // half of each weight, below 2^31
                const uint32_t a0 = __float2uint_rn(wt[0] * 2147483648.f), a1 = __float2uint_rn(wt[1] * 2147483648.f),
                               a2 = __float2uint_rn(wt[2] * 2147483648.f);
                const uint32_t s0 = q[0] + a0, s1 = q[32] + a1, s2 = q[64] + a2;
                q[0] = s0;
                q[32] = s1;
                q[64] = s2;
                if (s0 < a0 || s1 < a1 || s2 < a2) {
                    if (s0 < a0) atomicAdd(&carry[k0 + 1], 1u);
                    if (s1 < a1) atomicAdd(&carry[k0 + 2], 1u);
                    if (s2 < a2) atomicAdd(&carry[k0 + 3], 1u);
                }
            }
        });
    }
    // energy: FP64 warp sums, then the block's warps in a fixed order
    const double ew = warp_sum_d(0.5 * (double)e);
    if (lane == 0) s_e[w] = ew;
    __syncthreads();
    for (int b = w; b < n_bins; b += kLossTB / 32) {
        double v = 0.0;   // an integer below 2^53
#pragma unroll
        for (int q = 0; q < kLossTB / 32; q++) v += (double)s_hist[((size_t)q * rows + b + 1) * 32 + lane];
        v = warp_sum_d(v);
        if (lane == 0 && (v != 0.0 || carry[b + 1]))
            atomicAdd(&h_out[b], (v * kHistUnit + (double)carry[b + 1]) * inv_n);
    }
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int q = 0; q < kLossTB / 32; q++) v += s_e[q];
        if (v != 0.0) atomicAdd(U_out, v);
    }
}

// ---------------------------------------------------------- bonded (duals) --
struct Dual {
    float v, t;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.t + b.t}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.t - b.t}; }
__device__ __forceinline__ Dual operator-(Dual a) { return {-a.v, -a.t}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return {a.v * b.v, a.v * b.t + a.t * b.v}; }
__device__ __forceinline__ Dual operator*(float s, Dual a) { return {s * a.v, s * a.t}; }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    const float q = a.v / b.v;
    return {q, (a.t - q * b.t) / b.v};
}
__device__ __forceinline__ Dual dsqrt(Dual a) {
    const float s = sqrtf(a.v);
    return {s, 0.5f * a.t / s};
}
__device__ __forceinline__ Dual datan2(Dual y, Dual x) {
    return {atan2f(y.v, x.v), (x.v * y.t - y.v * x.t) / (x.v * x.v + y.v * y.v)};
}
__device__ __forceinline__ Dual dsin(Dual a) { return {sinf(a.v), cosf(a.v) * a.t}; }
__device__ __forceinline__ Dual dcos(Dual a) { return {cosf(a.v), -sinf(a.v) * a.t}; }
__device__ __forceinline__ Dual dmaxf(Dual a, float b) { return a.v > b ? a : Dual{b, 0.f}; }

struct D3 {
    Dual x, y, z;
};
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 operator-(D3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ D3 operator*(Dual s, D3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ Dual dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross(D3 a, D3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
// separation b - a (minimum image on the value, tangent passes through)
__device__ __forceinline__ D3 sep(const PhysDev& d, float4 a, float4 wa, float4 b, float4 wb) {
    return {{mimg_a(b.x - a.x, d.L, d.invL), wb.x - wa.x},
            {mimg_a(b.y - a.y, d.L, d.invL), wb.y - wa.y},
            {mimg_a(b.z - a.z, d.L, d.invL), wb.z - wa.z}};
}
__device__ __forceinline__ Dual cst(float v) { return {v, 0.f}; }

// MODE 0: bonded energy of the state into *U_out.  MODE 1: adjoint contributions.
// Every term's forces are F_q = g G_q: a scalar g that carries the constants
// (bond: -k (r - r0); angle: k (theta - theta0); dihedral: dV/dphi =
// -k n sin(n phi - phi0)) times directions G_q that depend on the positions
// only.  The constants' derivatives of the loss at this state are then
//   dL/dc = dt (dg/dc) sum_q w_q . G_q + le dE/dc     (c = r0 | theta0 | phi0, k)
// and go to the term's own FP64 accumulator (one thread per term: no atomics,
// the same order every run).
template <int MODE>
__global__ void __launch_bounds__(kAdjTB) k_adj_bonded(PhysDev d, const float4* __restrict__ po, AdjArgs a,
                                                       int hvp, double* U_out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nb = d.n_bonds, na = d.n_angles, nd = d.n_dih;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto W = [&](int orig) { return (MODE == 1 && hvp) ? a.wv[d.sorted_of_orig[orig]] : zero; };
    int n_at = 0, slot0 = 0;
    bool live = false;
    int at[4] = {0, 0, 0, 0};
    D3 G[4];
    Dual g = cst(0.f), E = cst(0.f);
    float dg_dc = 0.f, dg_dk = 0.f, dE_dc = 0.f, dE_dk = 0.f;
    if (t < nb) {
        live = true;
        const int4 ix = d.bond_idx[t];
        const float2 par = d.bond_par[t];
        at[0] = ix.x, at[1] = ix.y, n_at = 2, slot0 = 2 * t;
        const D3 r = sep(d, po[ix.x], W(ix.x), po[ix.y], W(ix.y));
        const Dual rr = dsqrt(dot(r, r));
        const Dual dr = rr - cst(par.x);
        G[1] = (cst(1.f) / rr) * r;   // F_j = -k (r - r0) r / |r|
        G[0] = -G[1];
        g = (-par.y) * dr;
        E = (0.5f * par.y) * (dr * dr);
        dg_dc = par.y, dg_dk = -dr.v;
        dE_dc = -par.y * dr.v, dE_dk = 0.5f * dr.v * dr.v;
    } else if (t < nb + na) {
        live = true;
        const int q = t - nb;
        const int4 ix = d.angle_idx[q];
        const float2 par = d.angle_par[q];
        at[0] = ix.x, at[1] = ix.y, at[2] = ix.z, n_at = 3, slot0 = 2 * nb + 3 * q;
        const D3 u = sep(d, po[ix.y], W(ix.y), po[ix.x], W(ix.x));   // x_i - x_j
        const D3 v = sep(d, po[ix.y], W(ix.y), po[ix.z], W(ix.z));   // x_k - x_j
        const Dual uu = dot(u, u), vv = dot(v, v);
        const Dual nu = dsqrt(uu), nv = dsqrt(vv);
        const D3 c = cross(u, v);
        const Dual sn = dsqrt(dot(c, c));
        const Dual cs = dot(u, v);
        const Dual th = datan2(sn, cs);
        const Dual dth = th - cst(par.x);
        const Dual inuv = cst(1.f) / (nu * nv);
        const Dual cosv = cs * inuv;
        const Dual is = cst(1.f) / dmaxf(sn * inuv, 1e-6f);
        G[0] = is * (inuv * v - (cosv / uu) * u);
        G[2] = is * (inuv * u - (cosv / vv) * v);
        G[1] = -(G[0] + G[2]);
        g = par.y * dth;
        E = (0.5f * par.y) * (dth * dth);
        dg_dc = -par.y, dg_dk = dth.v;
        dE_dc = -par.y * dth.v, dE_dk = 0.5f * dth.v * dth.v;
    } else if (t < nb + na + nd) {
        live = true;
        const int q = t - nb - na;
        const int4 ix = d.dih_idx[q];
        const float4 par = d.dih_par[q];
        at[0] = ix.x, at[1] = ix.y, at[2] = ix.z, at[3] = ix.w, n_at = 4, slot0 = 2 * nb + 3 * na + 4 * q;
        const D3 b1 = sep(d, po[ix.x], W(ix.x), po[ix.y], W(ix.y));
        const D3 b2 = sep(d, po[ix.y], W(ix.y), po[ix.z], W(ix.z));
        const D3 b3 = sep(d, po[ix.z], W(ix.z), po[ix.w], W(ix.w));
        const D3 m1 = cross(b1, b2), m2 = cross(b2, b3);
        const Dual m1m1 = dot(m1, m1), m2m2 = dot(m2, m2), b2b2 = dot(b2, b2);
        const Dual nb2 = dsqrt(b2b2);
        const Dual phi = datan2(nb2 * dot(b1, m2), dot(m1, m2));
        const Dual arg = par.z * phi - cst(par.x);
        const Dual sa = dsin(arg);
        const D3 hi = (nb2 / m1m1) * m1, hl = -((nb2 / m2m2) * m2);
        const Dual p = dot(b1, b2) / b2b2, r = dot(b3, b2) / b2b2;
        G[0] = hi;
        G[1] = -hi - p * hi + r * hl;
        G[2] = -hl + p * hi - r * hl;
        G[3] = hl;
        g = (-par.y * par.z) * sa;
        E = par.y * (cst(1.f) + dcos(arg));
        const float ca = cosf(arg.v);
        dg_dc = par.y * par.z * ca, dg_dk = -par.z * sa.v;
        dE_dc = par.y * sa.v, dE_dk = 1.f + ca;
    }
    // reductions
    double eu = 0.0;
    if (live) {
        if (MODE == 0) {
            eu = (double)E.v;
        } else {
            float sg = 0.f;   // sum_q w_q . G_q
            for (int q = 0; q < n_at; q++) {
                const float4 wq = W(at[q]);
                const D3 f = g * G[q];
                if (hvp) sg += wq.x * G[q].x.v + wq.y * G[q].y.v + wq.z * G[q].z.v;
                const float4 o = make_float4((hvp ? a.dt * f.x.t : 0.f) - a.le * f.x.v,
                                             (hvp ? a.dt * f.y.t : 0.f) - a.le * f.y.v,
                                             (hvp ? a.dt * f.z.t : 0.f) - a.le * f.z.v, 0.f);
                a.adj_term[d.bterm_pos[slot0 + q]] = o;
            }
            double2 acc = a.gterm[t];
            acc.x += (double)(a.dt * dg_dc * sg + a.le * dE_dc);
            acc.y += (double)(a.dt * dg_dk * sg + a.le * dE_dk);
            a.gterm[t] = acc;
        }
    }
    if (MODE == 0) {
        __shared__ double s_b[kAdjTB / 32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const double v0 = warp_sum_d(eu);
        if (lane == 0) s_b[w] = v0;
        __syncthreads();
        if (threadIdx.x == 0) {
            double v = 0.0;
            for (int q = 0; q < (int)(blockDim.x >> 5); q++) v += s_b[q];
            if (v != 0.0) atomicAdd(U_out, v);
        }
    }
}

// --------------------------------------------------------------- adjoint ---
// mu = lv + dt lx;  lv <- mu;  w = mu / m
__global__ void k_adj_prep(PhysDev d, AdjArgs a, float4* __restrict__ lam_v, float4* __restrict__ wv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const float4 lx = a.lam_x[i], lv = lam_v[i];
    const float im = d.vel[i].w;
    const float mx = lv.x + a.dt * lx.x, my = lv.y + a.dt * lx.y, mz = lv.z + a.dt * lx.z;
    lam_v[i] = make_float4(mx, my, mz, 0.f);
    wv[i] = make_float4(mx * im, my * im, mz * im, 0.f);
}

// LANES lanes (8 or 16, pair_lanes) per particle.  Every entry is evaluated
// (beyond r_c the switch and its derivatives are zero, beyond the last bin the
// staged occupancy error is), so a warp's lanes stay together.  The quotients of the per-type chain rule
// (sigma_ij = (s_a + s_b) / 2, eps_ij = sqrt(e_a e_b)) are a table per type
// pair.  The derivatives that land on the neighbour's type go to a column of
// the lane's own in shared memory ([2 types][32] per warp: no conflicts, no
// atomics; one type: registers), and are summed over the block in FP64.
// 8,192 particles on one B200: 55 us with per-thread arrays indexed by type
// (local memory) and four IEEE divisions an entry.
constexpr int kAdjPairTB = 128;
constexpr size_t kAdjPairStaticSmem = sizeof(float) * (LIMA_LOSS_MAX_BINS + 8);
constexpr size_t adj_pair_smem(int nt) {
    return sizeof(float4) * nt * nt + sizeof(float2) * (nt * nt + (nt * nt & 1)) +
           sizeof(float) * 32 * (kAdjPairTB / 32) * 2 * nt;
}
template <bool HVP, bool LOSS, typename ID, int LANES>
__global__ void __launch_bounds__(kAdjPairTB) k_adj_pair(PhysDev d, const float4* __restrict__ pos, AdjArgs a,
                                                         const double* __restrict__ hist_n,
                                                         const double* __restrict__ target) {
    extern __shared__ float4 s_dyn[];
    __shared__ float s_c[LIMA_LOSS_MAX_BINS + 8];   // occupancy error of bin b at b + 1, zero outside
    const int nt = a.n_types;
    // per type pair: (sigma^2, 4 eps, 1 / sigma, 0) and d eps_ij / d eps of i's and j's type
    float4* s_tab = s_dyn;
    float2* s_de = reinterpret_cast<float2*>(s_dyn + nt * nt);
    float* s_g = reinterpret_cast<float*>(s_de + nt * nt + (nt * nt & 1));   // [warps][2 nt][32]
    for (int q = threadIdx.x; q < nt * nt; q += blockDim.x) {
        const float2 t = d.lj_table[q];
        s_tab[q] = make_float4(t.x, t.y, rsqrtf(t.x), 0.f);
        const float ei = a.par[nt + q / nt], ej = a.par[nt + q % nt], e = 0.25f * t.y;
        s_de[q] = make_float2(ei > 0.f ? e / (2.f * ei) : 0.f, ej > 0.f ? e / (2.f * ej) : 0.f);
    }
    if (LOSS)
        for (int q = threadIdx.x; q < LIMA_LOSS_MAX_BINS + 8; q += blockDim.x)
            s_c[q] = q >= 1 && q <= a.n_bins ? (float)(hist_n[q - 1] - target[q - 1]) : 0.f;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool one = nt == 1;
    float* mine = s_g + (size_t)w * 2 * nt * 32 + lane;   // the lane's column
    for (int q = 0; q < 2 * nt; q++) mine[q * 32] = 0.f;
    __syncthreads();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int g = threadIdx.x % LANES;
    float hx = 0.f, hy = 0.f, hz = 0.f;   // dt * sum J (w_i - w_j)  (dt applied at the end)
    float fx = 0.f, fy = 0.f, fz = 0.f;   // LJ force on i
    float rx = 0.f, ry = 0.f, rz = 0.f;   // sum G(r) d
    float gs_a = 0.f, ge_a = 0.f;         // parameter derivatives landing on i's type
    float gs_1 = 0.f, ge_1 = 0.f;         // on j's type, where there is one type
    int ti = 0;
    if (i < d.n) {
        const float4 pi = pos[i];
        ti = __float_as_int(pi.w);
        const float4 wi = HVP ? a.wv[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const int cnt = (int)d.nl_cnt[i];
        const bool rdf = LOSS && a.lr != 0.f;
        const float hdt = 0.5f * a.dt, hle = 0.5f * a.le;
        const int kmax = a.n_bins + 1;
        for_entries<LANES, ID>(d, pos, i, g, cnt, [&](uint32_t j, float4 pj) {
            const float dx = mimg_add(pi.x - pj.x, d.L, d.invL), dy = mimg_add(pi.y - pj.y, d.L, d.invL),
                        dz = mimg_add(pi.z - pj.z, d.L, d.invL);
            const float r2 = dx * dx + dy * dy + dz * dz;
            const int tj = __float_as_int(pj.w), tt = ti * nt + tj;
            const float4 tab = s_tab[tt];
            const float e4 = tab.y;   // 4 eps_ij
            const LJ1 l = lj1(d, r2, tab.x, tab.z);
            float dsig = 0.f, deps4 = 0.f;   // d/d sigma_ij and d/d (4 eps_ij) of this visit
            if (HVP) {
                const float4 wj = __ldg(a.wv + j);
                const float ux = wi.x - wj.x, uy = wi.y - wj.y, uz = wi.z - wj.z;
                const float du = dx * ux + dy * uy + dz * uz;
                const float c1 = e4 * l.f, c2 = 2.f * e4 * l.fp * du;
                hx += c1 * ux + c2 * dx;
                hy += c1 * uy + c2 * dy;
                hz += c1 * uz + c2 * dz;
                // half of dt (w_i - w_j) . dF_i/dtheta (the other half comes from j's visit)
                dsig += hdt * du * e4 * l.df_ds;
                deps4 += hdt * du * l.f;
            }
            if (LOSS) {
                const float f = e4 * l.f;
                fx += f * dx;
                fy += f * dy;
                fz += f * dz;
                dsig += hle * e4 * l.dph_ds;
                deps4 += hle * l.ph;
                if (rdf) {
                    const float r = sqrtf(r2);
                    int k0;
                    float wt[3], dw[3];
                    bspline3(r, a.inv_dr, k0, wt, dw);
                    k0 = min(k0, kmax);   // past the support: zeros
                    const float* c = s_c + k0 + 1;
                    const float G = quot_newton(c[0] * dw[0] + c[1] * dw[1] + c[2] * dw[2], r);
                    rx += G * dx;
                    ry += G * dy;
                    rz += G * dz;
                }
            }
            // chain to the per-type parameters
            const float2 de = s_de[tt];
            const float hs = 0.5f * dsig, d4 = 4.f * deps4;   // d/d eps_ij
            gs_a += hs;
            ge_a += d4 * de.x;
            if (one) {
                gs_1 += hs;
                ge_1 += d4 * de.y;
            } else {
                mine[tj * 32] += hs;
                mine[(nt + tj) * 32] += d4 * de.y;
            }
        });
        mine[ti * 32] += gs_a + gs_1;   // one type: gs_1 is its other half
        mine[(nt + ti) * 32] += ge_a + ge_1;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        hx += __shfl_xor_sync(0xffffffffu, hx, o);
        hy += __shfl_xor_sync(0xffffffffu, hy, o);
        hz += __shfl_xor_sync(0xffffffffu, hz, o);
        fx += __shfl_xor_sync(0xffffffffu, fx, o);
        fy += __shfl_xor_sync(0xffffffffu, fy, o);
        fz += __shfl_xor_sync(0xffffffffu, fz, o);
        rx += __shfl_xor_sync(0xffffffffu, rx, o);
        ry += __shfl_xor_sync(0xffffffffu, ry, o);
        rz += __shfl_xor_sync(0xffffffffu, rz, o);
    }
    if (i < d.n && g == 0) {
        float bx = 0.f, by = 0.f, bz = 0.f;
        const uint32_t oi = d.orig_of_sorted[i];
        if (oi < (uint32_t)d.n_cp) {
            const uint32_t q1 = d.bterm_off[oi + 1];
#pragma unroll 4
            for (uint32_t q = d.bterm_off[oi]; q < q1; q++) {
                const float4 tf = a.adj_term[q];
                bx += tf.x;
                by += tf.y;
                bz += tf.z;
            }
        }
        float4 lx = a.lam_x[i];
        lx.x += a.dt * hx - a.le * fx + a.lr * rx + bx;
        lx.y += a.dt * hy - a.le * fy + a.lr * ry + by;
        lx.z += a.dt * hz - a.le * fz + a.lr * rz + bz;
        a.lam_x[i] = lx;
    }
    __syncthreads();
    // parameter derivatives: the block's lanes in FP64, then global
    for (int q = w; q < 2 * nt; q += kAdjPairTB / 32) {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < kAdjPairTB / 32; k++) v += (double)s_g[((size_t)k * 2 * nt + q) * 32 + lane];
        v = warp_sum_d(v);
        if (lane == 0 && v != 0.0) atomicAdd(&a.gtheta[q], v);
    }
}

// ---------------------------------------------------------- state moves ---
__global__ void k_save(PhysDev d, int cur, float4* __restrict__ x, float4* __restrict__ v) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.n) return;
    const uint32_t o = d.orig_of_sorted[k];
    x[o] = d.pos[cur][k];
    v[o] = d.vel[k];
}

// state in orig order; the next rebuild sorts it
__global__ void k_restore(PhysDev d, int cur, const float4* __restrict__ x, const float4* __restrict__ v) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= d.n) return;
    const float4 p = x[o];
    d.pos[cur][o] = p;
    d.vel[o] = v[o];
    d.orig_of_sorted[o] = (uint32_t)o;
    d.sorted_of_orig[o] = (uint32_t)o;
    if (o < d.n_cp) d.pos_orig[cur][o] = p;
}

__global__ void k_to_sorted(PhysDev d, const float4* __restrict__ in, float4* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.n) out[k] = in[d.orig_of_sorted[k]];
}

__global__ void k_to_orig(PhysDev d, const float4* __restrict__ in, float4* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.n) out[d.orig_of_sorted[k]] = in[k];
}

template <typename T>
T* grow(std::vector<void*>& allocs, size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) return nullptr;
    allocs.push_back(p);
    return static_cast<T*>(p);
}

bool ensure(const PhysDev& d, AdjBuffers& A, std::vector<void*>& allocs, int n_ckpt, int n_seg, int n_steps,
            int n_bins) {
    const size_t n = (size_t)d.n, np = (size_t)d.n_pad, ncp = (size_t)std::max(d.n_cp, 1);
    if (!A.lam_x) {
        A.lam_x = grow<float4>(allocs, np);
        A.lam_v = grow<float4>(allocs, np);
        A.wv = grow<float4>(allocs, np);
        A.lam_xo = grow<float4>(allocs, n);
        A.lam_vo = grow<float4>(allocs, n);
        A.adj_term = grow<float4>(allocs, (size_t)std::max(d.n_term_slots, 1));
        A.gtheta = grow<double>(allocs, 2 * kMaxTypes + kParKinds);
        A.par = grow<float>(allocs, 2 * kMaxTypes + kParKinds);
        A.cap_terms = std::max(d.n_bonds + d.n_angles + d.n_dih, 1);
        A.gterm = grow<double2>(allocs, (size_t)A.cap_terms);
        if (!A.lam_x || !A.lam_v || !A.wv || !A.lam_xo || !A.lam_vo || !A.adj_term || !A.gtheta || !A.par ||
            !A.gterm)
            return false;
    }
    if (n_ckpt > A.cap_ckpt) {
        A.ck_x = grow<float4>(allocs, n * n_ckpt);
        A.ck_v = grow<float4>(allocs, n * n_ckpt);
        if (!A.ck_x || !A.ck_v) return false;
        A.cap_ckpt = n_ckpt;
    }
    if (n_seg > A.cap_seg) {
        A.seg_x = grow<float4>(allocs, np * n_seg);
        A.seg_xo = grow<float4>(allocs, ncp * n_seg);
        if (!A.seg_x || !A.seg_xo) return false;
        A.cap_seg = n_seg;
    }
    if (n_steps > A.cap_steps || n_bins > A.cap_bins) {
        const int st = std::max(n_steps, A.cap_steps), nb = std::max(n_bins, A.cap_bins);
        A.U = grow<double>(allocs, (size_t)st + 1);
        A.hist = grow<double>(allocs, ((size_t)st + 1) * nb);
        A.target = grow<double>(allocs, nb);
        if (!A.U || !A.hist || !A.target) return false;
        A.cap_steps = st;
        A.cap_bins = nb;
    }
    return true;
}

int read_err(const PhysDev& d, cudaStream_t s) {
    int h = 0;
    cudaMemcpyAsync(&h, d.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    return h;
}

}  // namespace

// ------------------------------------------------------------- parameters --
namespace {
// Groups the loaded terms of one kind into types: the distinct constant sets
// (c, k, n) in ascending order; type_of[t] is term t's type.
void group_terms(const std::vector<float4>& terms, std::vector<int>& type_of, std::vector<float4>& type0) {
    auto less = [](const float4& a, const float4& b) {
        if (a.x != b.x) return a.x < b.x;
        if (a.y != b.y) return a.y < b.y;
        return a.z < b.z;
    };
    type0 = terms;
    std::sort(type0.begin(), type0.end(), less);
    type0.erase(std::unique(type0.begin(), type0.end(),
                            [](const float4& a, const float4& b) { return a.x == b.x && a.y == b.y && a.z == b.z; }),
                type0.end());
    type_of.resize(terms.size());
    for (size_t t = 0; t < terms.size(); t++)
        type_of[t] = (int)(std::lower_bound(type0.begin(), type0.end(), terms[t], less) - type0.begin());
}
}  // namespace

void phys_params_init(const PhysDev& d, const lima_forcefield& ff, PhysParams& pp, cudaStream_t s) {
    pp.n_types = d.n_types;
    pp.sigma.resize(d.n_types);
    pp.epsilon.resize(d.n_types);
    for (int t = 0; t < d.n_types; t++) {
        pp.sigma[t] = ff.particle_parameters[t].sigma;
        pp.epsilon[t] = ff.particle_parameters[t].epsilon;
    }
    pp.scale[0] = pp.scale[1] = pp.scale[2] = 1.0;
    pp.bond0.resize(d.n_bonds);
    pp.angle0.resize(d.n_angles);
    pp.dih0.resize(d.n_dih);
    if (d.n_bonds) cudaMemcpyAsync(pp.bond0.data(), d.bond_par, sizeof(float2) * d.n_bonds, cudaMemcpyDeviceToHost, s);
    if (d.n_angles)
        cudaMemcpyAsync(pp.angle0.data(), d.angle_par, sizeof(float2) * d.n_angles, cudaMemcpyDeviceToHost, s);
    if (d.n_dih) cudaMemcpyAsync(pp.dih0.data(), d.dih_par, sizeof(float4) * d.n_dih, cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    std::vector<float4> terms[kParKinds];
    for (const float2& b : pp.bond0) terms[kParBond].push_back(make_float4(b.x, b.y, 0.f, 0.f));
    for (const float2& a : pp.angle0) terms[kParAngle].push_back(make_float4(a.x, a.y, 0.f, 0.f));
    for (const float4& q : pp.dih0) terms[kParDihedral].push_back(make_float4(q.x, q.y, q.z, 0.f));
    for (int k = 0; k < kParKinds; k++) {
        group_terms(terms[k], pp.type_of[k], pp.type0[k]);
        pp.tc[k].resize(pp.type0[k].size());
        pp.tk[k].resize(pp.type0[k].size());
        for (size_t q = 0; q < pp.type0[k].size(); q++) {
            pp.tc[k][q] = pp.type0[k][q].x;
            pp.tk[k][q] = pp.type0[k][q].y;
        }
    }
}

void phys_params_get(const PhysParams& pp, double* theta) {
    const int nt = pp.n_types;
    for (int t = 0; t < nt; t++) {
        theta[t] = pp.sigma[t];
        theta[nt + t] = pp.epsilon[t];
    }
    for (int k = 0; k < kParKinds; k++) theta[2 * nt + k] = pp.scale[k];
    double* o = theta + 2 * nt + kParKinds;
    for (int k = 0; k < kParKinds; k++)
        for (size_t q = 0; q < pp.tc[k].size(); q++) {
            *o++ = pp.tc[k][q];
            *o++ = pp.tk[k][q];
        }
}

int phys_params_set(PhysDev& d, PhysParams& pp, const double* theta, std::string& msg, cudaStream_t s) {
    const int nt = pp.n_types;
    for (int t = 0; t < nt; t++)
        if (!(theta[t] > 0.0) || !(theta[nt + t] >= 0.0) || !std::isfinite(theta[t]) || !std::isfinite(theta[nt + t])) {
            msg = "sigma must be positive and epsilon non-negative (finite)";
            return LIMA_ERR_ARGUMENT;
        }
    for (int k = 0; k < kParKinds; k++)
        if (!(theta[2 * nt + k] >= 0.0) || !std::isfinite(theta[2 * nt + k])) {
            msg = "bonded scales must be finite and non-negative";
            return LIMA_ERR_ARGUMENT;
        }
    const double* tt = theta + 2 * nt + kParKinds;
    for (int k = 0, o = 0; k < kParKinds; k++)
        for (size_t q = 0; q < pp.tc[k].size(); q++, o += 2)
            if (!std::isfinite(tt[o]) || !std::isfinite(tt[o + 1]) || !(tt[o + 1] >= 0.0) ||
                (k == kParBond && !(tt[o] > 0.0))) {
                msg = "bonded type constants must be finite, force constants non-negative and bond lengths positive";
                return LIMA_ERR_ARGUMENT;
            }
    for (int t = 0; t < nt; t++) {
        pp.sigma[t] = theta[t];
        pp.epsilon[t] = theta[nt + t];
    }
    for (int k = 0; k < kParKinds; k++) pp.scale[k] = theta[2 * nt + k];
    for (int k = 0, o = 0; k < kParKinds; k++)
        for (size_t q = 0; q < pp.tc[k].size(); q++, o += 2) {
            pp.tc[k][q] = tt[o];
            pp.tk[k][q] = tt[o + 1];
        }
    std::vector<float2> tab((size_t)nt * nt);
    for (int a = 0; a < nt; a++)
        for (int b = 0; b < nt; b++) {
            const double sg = 0.5 * (pp.sigma[a] + pp.sigma[b]);
            const double ep = std::sqrt(pp.epsilon[a] * pp.epsilon[b]);
            tab[a * nt + b] = make_float2((float)(sg * sg), (float)(4.0 * ep));
        }
    // every term takes its type's constants; the force constant times the kind's scale
    std::vector<float2> bp(pp.bond0), ap(pp.angle0);
    std::vector<float4> dp(pp.dih0);
    for (size_t t = 0; t < bp.size(); t++) {
        const int q = pp.type_of[kParBond][t];
        bp[t] = make_float2((float)pp.tc[kParBond][q], (float)(pp.tk[kParBond][q] * pp.scale[kParBond]));
    }
    for (size_t t = 0; t < ap.size(); t++) {
        const int q = pp.type_of[kParAngle][t];
        ap[t] = make_float2((float)pp.tc[kParAngle][q], (float)(pp.tk[kParAngle][q] * pp.scale[kParAngle]));
    }
    for (size_t t = 0; t < dp.size(); t++) {
        const int q = pp.type_of[kParDihedral][t];
        dp[t].x = (float)pp.tc[kParDihedral][q];
        dp[t].y = (float)(pp.tk[kParDihedral][q] * pp.scale[kParDihedral]);
    }
    cudaMemcpyAsync(d.lj_table, tab.data(), sizeof(float2) * tab.size(), cudaMemcpyHostToDevice, s);
    if (!bp.empty()) cudaMemcpyAsync(d.bond_par, bp.data(), sizeof(float2) * bp.size(), cudaMemcpyHostToDevice, s);
    if (!ap.empty()) cudaMemcpyAsync(d.angle_par, ap.data(), sizeof(float2) * ap.size(), cudaMemcpyHostToDevice, s);
    if (!dp.empty()) cudaMemcpyAsync(d.dih_par, dp.data(), sizeof(float4) * dp.size(), cudaMemcpyHostToDevice, s);
    cudaStreamSynchronize(s);
    return cudaGetLastError() == cudaSuccess ? LIMA_OK : LIMA_ERR_CUDA;
}

// ------------------------------------------------------------------ passes --
namespace {

// Lanes that share one particle's list in the adjoint pair kernel: 8, and 16
// in boxes whose 8-lane grid leaves most of an SM's warps unfilled.  A 50-step
// gradient of 1,948 particles took 6.44 ms with 8, 5.82 with 16, 5.88 with 32;
// 40 steps of 5,040 particles 5.54, 5.25, 5.82; 200 steps of 8,192 particles
// 26.3, 27.6, 30.8 (with the loss kernel on as many lanes).  The loss kernel
// keeps 8: more lanes are more columns of occupancies to clear and sum (200
// steps of 8,192 particles: 11.5 ms with 8, 14.1 with 16).  The line lies between
// 5,040 and 8,192; no size between them was measured, nor another cutoff, which
// changes the list a lane walks.
int pair_lanes(int n) { return n < 6144 ? 16 : kGroup; }

struct Runner {
    PhysDev d;           // copy with fixed-period list semantics (stale -> error)
    AdjBuffers& A;
    cudaStream_t s;
    int n_bins;
    float inv_dr, supp2;
    int tb = 256;
    int blocks_n() const { return (d.n + tb - 1) / tb; }
    int blocks_pair(int threads, int lanes) const { return (int)(((size_t)d.n * lanes + threads - 1) / threads); }
    int blocks_terms() const { return std::max(1, (d.n_bonds + d.n_angles + d.n_dih + kAdjTB - 1) / kAdjTB); }

    void save(int cur, int k) { k_save<<<blocks_n(), tb, 0, s>>>(d, cur, A.ck_x + (size_t)k * d.n, A.ck_v + (size_t)k * d.n); }
    void restore(int cur, int k) {
        k_restore<<<blocks_n(), tb, 0, s>>>(d, cur, A.ck_x + (size_t)k * d.n, A.ck_v + (size_t)k * d.n);
        phys_rebuild(d, cur, s);
    }
    // energy and occupancies of the state in parity cur -> U[n], hist[n]
    void loss_pass(int cur, const float4* pos, const float4* po, int n) {
        const size_t smem = loss_smem(n_bins);
        auto run = [&](auto kernel) {
            allow_smem(kernel, smem, kLossStaticSmem, loss_smem(LIMA_LOSS_MAX_BINS));
            kernel<<<blocks_pair(kLossTB, kGroup), kLossTB, smem, s>>>(d, pos, n_bins, inv_dr, supp2, 1.0 / d.n, A.U + n,
                                                               A.hist + (size_t)n * n_bins);
        };
        if (d.nl16) run(k_loss_pairs<uint16_t>);
        else run(k_loss_pairs<uint32_t>);
        if (d.n_bonds + d.n_angles + d.n_dih > 0) {
            AdjArgs a{};
            k_adj_bonded<0><<<blocks_terms(), kAdjTB, 0, s>>>(d, po, a, 0, A.U + n);
        }
        (void)cur;
    }
    // one adjoint pair pass over the state xs (hist_n: its occupancies, with a loss term)
    template <bool HVP, bool LOSS>
    void adj_pair(const float4* xs, const AdjArgs& a, const double* hist_n) {
        const size_t smem = adj_pair_smem(a.n_types);
        auto run = [&](auto kernel) {
            allow_smem(kernel, smem, kAdjPairStaticSmem, adj_pair_smem(kMaxTypes));
            kernel<<<blocks_pair(kAdjPairTB, pair_lanes(d.n)), kAdjPairTB, smem, s>>>(d, xs, a, hist_n, A.target);
        };
        if (pair_lanes(d.n) == 16) {
            if (d.nl16) run(k_adj_pair<HVP, LOSS, uint16_t, 16>);
            else run(k_adj_pair<HVP, LOSS, uint32_t, 16>);
        } else {
            if (d.nl16) run(k_adj_pair<HVP, LOSS, uint16_t, kGroup>);
            else run(k_adj_pair<HVP, LOSS, uint32_t, kGroup>);
        }
    }
    void adj_bonded(const float4* xo, const AdjArgs& a, int hvp) {
        if (d.n_bonds + d.n_angles + d.n_dih > 0) k_adj_bonded<1><<<blocks_terms(), kAdjTB, 0, s>>>(d, xo, a, hvp, nullptr);
    }
};

double loss_of(const std::vector<double>& U, const std::vector<double>& H, const std::vector<double>& target, int T,
               int n_bins, int n, double we, double wr) {
    double L = 0.0;
    for (int k = 1; k <= T; k++) {
        double r = 0.0;
        for (int b = 0; b < n_bins; b++) {
            const double c = H[(size_t)k * n_bins + b] - (target.empty() ? 0.0 : target[b]);
            r += c * c;
        }
        L += we * U[k] / n + wr * r;
    }
    return L / T;
}

}  // namespace

int adj_rdf(const PhysDev& d, int cur, AdjBuffers& A, std::vector<void*>& allocs, int n_bins, float r_max, double* h,
            cudaStream_t s, std::string& msg) {
    if (n_bins < 1 || n_bins > LIMA_LOSS_MAX_BINS || !(r_max > 0.f)) {
        msg = "need 1 <= n_bins <= LIMA_LOSS_MAX_BINS and r_max > 0";
        return LIMA_ERR_ARGUMENT;
    }
    const float dr = r_max / n_bins;
    if (r_max + dr > d.rc * (1.f + 1e-6f)) {
        msg = "r_max + r_max/n_bins must not exceed the cutoff";
        return LIMA_ERR_ARGUMENT;
    }
    if (!ensure(d, A, allocs, 1, 1, 1, n_bins)) {
        msg = "cudaMalloc failed for the loss buffers";
        return LIMA_ERR_CUDA;
    }
    Runner R{d, A, s, n_bins, 1.f / dr, (r_max + dr) * (r_max + dr)};
    cudaMemsetAsync(A.hist, 0, sizeof(double) * n_bins, s);
    cudaMemsetAsync(A.U, 0, sizeof(double), s);
    R.loss_pass(cur, d.pos[cur], d.pos_orig[cur], 0);
    cudaMemcpyAsync(h, A.hist, sizeof(double) * n_bins, cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    return cudaGetLastError() == cudaSuccess ? LIMA_OK : LIMA_ERR_CUDA;
}

int adj_run(const PhysDev& d0, int cur, const PhysParams& pp, AdjBuffers& A, std::vector<void*>& allocs,
            const lima_loss_spec& spec, double* loss, double* grad, cudaStream_t s, std::string& msg) {
    const int T = spec.n_steps;
    if (T < 1 || spec.checkpoint_every < 1 || spec.n_bins < 1 || spec.n_bins > LIMA_LOSS_MAX_BINS ||
        !(spec.r_max > 0.f) || !std::isfinite(spec.w_energy) || !std::isfinite(spec.w_rdf)) {
        msg = "loss spec: need n_steps >= 1, checkpoint_every >= 1, 1 <= n_bins <= 128, r_max > 0, finite weights";
        return LIMA_ERR_ARGUMENT;
    }
    if (spec.w_rdf != 0.0 && !spec.rdf_target) {
        msg = "loss spec: rdf_target is required when w_rdf != 0";
        return LIMA_ERR_ARGUMENT;
    }
    const int nb = spec.n_bins;
    const float dr = spec.r_max / nb;
    if (spec.r_max + dr > d0.rc * (1.f + 1e-6f)) {
        msg = "loss spec: r_max + r_max/n_bins must not exceed the cutoff";
        return LIMA_ERR_ARGUMENT;
    }
    const int C = std::min(spec.checkpoint_every, T);
    const int K = (T + C - 1) / C;
    if (!ensure(d0, A, allocs, K, C + 1, T, nb)) {
        msg = "cudaMalloc failed for the adjoint buffers";
        return LIMA_ERR_CUDA;
    }
    PhysDev d = d0;
    d.dynamic_list = 0;
    Runner R{d, A, s, nb, 1.f / dr, (spec.r_max + dr) * (spec.r_max + dr)};
    std::vector<double> target(nb, 0.0);
    if (spec.rdf_target) target.assign(spec.rdf_target, spec.rdf_target + nb);
    cudaMemcpyAsync(A.target, target.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(A.U, 0, sizeof(double) * (T + 1), s);
    cudaMemsetAsync(A.hist, 0, sizeof(double) * (size_t)(T + 1) * nb, s);
    cudaMemsetAsync(A.gtheta, 0, sizeof(double) * (2 * kMaxTypes + kParKinds), s);
    cudaMemsetAsync(A.gterm, 0, sizeof(double2) * A.cap_terms, s);
    const int nt = pp.n_types;
    std::vector<float> par(2 * nt + kParKinds);
    for (int t = 0; t < nt; t++) {
        par[t] = (float)pp.sigma[t];
        par[nt + t] = (float)pp.epsilon[t];
    }
    for (int k = 0; k < kParKinds; k++) par[2 * nt + k] = (float)pp.scale[k];
    cudaMemcpyAsync(A.par, par.data(), sizeof(float) * par.size(), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(d.err, 0, sizeof(int), s);

    const int start_cur = cur;
    // the first launch or copy that failed, for the error message
    const char* fail_at = nullptr;
    cudaError_t fail_err = cudaSuccess;
    auto note = [&](const char* where) {
        if (fail_at) return;
        const cudaError_t e = cudaPeekAtLastError();
        if (e != cudaSuccess) {
            fail_at = where;
            fail_err = e;
        }
    };
    note("set-up copies");
    // forward: checkpoints at the start of every segment (re-sorted from orig
    // order there, so a recomputation reproduces the trajectory bit for bit)
    R.save(cur, 0);
    note("checkpoint save");
    for (int k = 0; k < K; k++) {
        const bool last = k == K - 1;
        if (grad && last) break;   // the backward pass recomputes the last segment anyway
        R.restore(cur, k);
        note("checkpoint restore and list rebuild");
        const int n0 = k * C, len = std::min(C, T - n0);
        for (int q = 0; q < len; q++) {
            if (q > 0 && q % kListEpoch == 0) phys_rebuild_inplace(d, d.pos[cur], s);
            note("in-place list rebuild");
            phys_step_kernels(d, cur, s, false);
            note("forward step kernels");
            cur ^= 1;
            if (!grad) R.loss_pass(cur, d.pos[cur], d.pos_orig[cur], n0 + q + 1);
            note("loss pass");
        }
        if (!last) R.save(cur, k + 1);
    }
    const double we = spec.w_energy, wr = spec.w_rdf;
    const float le = (float)(we / ((double)d.n * T)), lr = (float)(2.0 * wr / ((double)d.n * T));
    if (grad) {
        cudaMemsetAsync(A.lam_xo, 0, sizeof(float4) * d.n, s);
        cudaMemsetAsync(A.lam_vo, 0, sizeof(float4) * d.n, s);
        cudaMemsetAsync(A.lam_x, 0, sizeof(float4) * d.n_pad, s);
        cudaMemsetAsync(A.lam_v, 0, sizeof(float4) * d.n_pad, s);
        cudaMemsetAsync(A.wv, 0, sizeof(float4) * d.n_pad, s);
        AdjArgs a{};
        a.dt = (float)d.dt;
        a.inv_dr = R.inv_dr;
        a.supp2 = R.supp2;
        a.n_bins = nb;
        a.n_types = nt;
        a.lam_x = A.lam_x;
        a.wv = A.wv;
        a.adj_term = A.adj_term;
        a.par = A.par;
        a.gtheta = A.gtheta;
        a.gterm = A.gterm;
        for (int k = K - 1; k >= 0; k--) {
            const int n0 = k * C, len = std::min(C, T - n0);
            R.restore(cur, k);
            // recompute the segment, keeping every state and its loss terms
            cudaMemcpyAsync(A.seg_x, d.pos[cur], sizeof(float4) * d.n_pad, cudaMemcpyDeviceToDevice, s);
            if (d.n_cp)
                cudaMemcpyAsync(A.seg_xo, d.pos_orig[cur], sizeof(float4) * d.n_cp, cudaMemcpyDeviceToDevice, s);
            for (int q = 0; q < len; q++) {
                if (q > 0 && q % kListEpoch == 0) phys_rebuild_inplace(d, d.pos[cur], s);
                phys_step_kernels(d, cur, s, false);
                cur ^= 1;
                float4* xs = A.seg_x + (size_t)(q + 1) * d.n_pad;
                float4* xo = A.seg_xo + (size_t)(q + 1) * std::max(d.n_cp, 1);
                cudaMemcpyAsync(xs, d.pos[cur], sizeof(float4) * d.n_pad, cudaMemcpyDeviceToDevice, s);
                if (d.n_cp) cudaMemcpyAsync(xo, d.pos_orig[cur], sizeof(float4) * d.n_cp, cudaMemcpyDeviceToDevice, s);
                R.loss_pass(cur, xs, xo, n0 + q + 1);
            }
            k_to_sorted<<<R.blocks_n(), R.tb, 0, s>>>(d, A.lam_xo, A.lam_x);
            k_to_sorted<<<R.blocks_n(), R.tb, 0, s>>>(d, A.lam_vo, A.lam_v);
            // loss term of the segment's last state
            {
                const int q = len;
                a.le = le;
                a.lr = lr;
                const float4* xs = A.seg_x + (size_t)q * d.n_pad;
                const float4* xo = A.seg_xo + (size_t)q * std::max(d.n_cp, 1);
                R.adj_bonded(xo, a, 0);
                R.adj_pair<false, true>(xs, a, A.hist + (size_t)(n0 + q) * nb);
            }
            int epoch = (len - 1) / kListEpoch;   // the list built last
            for (int q = len - 1; q >= 0; q--) {
                if (q / kListEpoch != epoch) {
                    epoch = q / kListEpoch;
                    phys_rebuild_inplace(d, A.seg_x + (size_t)epoch * kListEpoch * d.n_pad, s);
                }
                const bool has_loss = q >= 1;
                a.le = has_loss ? le : 0.f;
                a.lr = has_loss ? lr : 0.f;
                const float4* xs = A.seg_x + (size_t)q * d.n_pad;
                const float4* xo = A.seg_xo + (size_t)q * std::max(d.n_cp, 1);
                k_adj_prep<<<R.blocks_n(), R.tb, 0, s>>>(d, a, A.lam_v, A.wv);
                R.adj_bonded(xo, a, 1);
                if (has_loss)
                    R.adj_pair<true, true>(xs, a, A.hist + (size_t)(n0 + q) * nb);
                else
                    R.adj_pair<true, false>(xs, a, nullptr);
            }
            k_to_orig<<<R.blocks_n(), R.tb, 0, s>>>(d, A.lam_x, A.lam_xo);
            k_to_orig<<<R.blocks_n(), R.tb, 0, s>>>(d, A.lam_v, A.lam_vo);
        }
    }
    // loss value
    std::vector<double> U(T + 1), H((size_t)(T + 1) * nb);
    cudaMemcpyAsync(U.data(), A.U, sizeof(double) * (T + 1), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(H.data(), A.hist, sizeof(double) * H.size(), cudaMemcpyDeviceToHost, s);
    std::vector<double> g(2 * nt, 0.0);
    const int n_terms = d.n_bonds + d.n_angles + d.n_dih;
    std::vector<double2> gt((size_t)n_terms);
    if (grad) {
        cudaMemcpyAsync(g.data(), A.gtheta, sizeof(double) * g.size(), cudaMemcpyDeviceToHost, s);
        if (n_terms) cudaMemcpyAsync(gt.data(), A.gterm, sizeof(double2) * n_terms, cudaMemcpyDeviceToHost, s);
    }
    const int err = read_err(d, s);
    // leave the state as found: restore the first checkpoint into the starting parity
    if (cur != start_cur) cur = start_cur;
    R.restore(cur, 0);
    cudaStreamSynchronize(s);
    note("the passes");
    const cudaError_t last_err = cudaGetLastError();
    if (fail_at || last_err != cudaSuccess) {
        msg = std::string("CUDA error in the loss / adjoint passes (") + (fail_at ? fail_at : "the passes") + "): " +
              cudaGetErrorString(fail_at ? fail_err : last_err);
        return LIMA_ERR_CUDA;
    }
    if (err) {
        cudaMemsetAsync(d.err, 0, sizeof(int), s);
        cudaStreamSynchronize(s);
        msg = (err & ERR_BIT_LIST_STALE) ? "pair list went stale inside a checkpoint segment (raise skin or lower "
                                           "checkpoint_every)"
                                         : "device error during the loss / adjoint passes";
        return LIMA_ERR_NUMERIC;
    }
    *loss = loss_of(U, H, target, T, nb, d.n, we, wr);
    if (grad) {
        for (size_t q = 0; q < g.size(); q++) grad[q] = g[q];
        // bonded constants: the terms' derivatives summed per type in term
        // order; a term's force constant is s_kind * k_type
        double* gs = grad + 2 * nt;
        double* gty = gs + kParKinds;
        for (int q = 0; q < kParKinds + 2 * pp.n_term_types(); q++) gs[q] = 0.0;
        const int base[kParKinds] = {0, d.n_bonds, d.n_bonds + d.n_angles};
        const int cnt[kParKinds] = {d.n_bonds, d.n_angles, d.n_dih};
        for (int k = 0, off = 0; k < kParKinds; off += 2 * (int)pp.tc[k].size(), k++)
            for (int t = 0; t < cnt[k]; t++) {
                const double2 v = gt[base[k] + t];
                const int q = pp.type_of[k][t];
                gs[k] += v.y * pp.tk[k][q];
                gty[off + 2 * q] += v.x;
                gty[off + 2 * q + 1] += v.y * pp.scale[k];
            }
    }
    return LIMA_OK;
}

}  // namespace lima
