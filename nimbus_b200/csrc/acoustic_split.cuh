// Two-launch acoustic substep, templated on the precision policy of
// acoustic_fused.cuh; one thread per cell (grid-stride), marching along x, or
// four vertically adjacent cells per thread (from kQuadCells on):
//   split_continuity_eos : retained mass flux from the old state, continuity,
//                          rho forward Euler, EOS; new rho to a ping-pong
//                          buffer, p in place.
//   split_momentum       : u,v,w forward Euler from the new pressure gradient,
//                          written to ping-pong buffers.
// No shared memory and no barriers: neighbour reuse comes from L1/L2 and
// latency is hidden by full occupancy.  It moves 84 B/cell (u,v,w are read
// twice, the new rho/p written then re-read) against the fused form's
// 64 B/cell, but issues fewer instructions per cell; the autotuner picks
// between the two per grid shape.
#pragma once

#include "acoustic_fused.cuh"
#include "acoustic_kernels.cuh"

namespace nimbus
{

// Retained-flux update from an already loaded slot value; returns the slot's
// new value.  Reference policy: the FP64 weighted sum rounded once to the FP32
// slot (fused_accumulate); FP32 policy: one FMA (retain_flux_f32).  With store
// the slot starts from zero -- the first substep of a large step writes
// instead of accumulating, bit-identical to accumulating into a zeroed slot
// (the 0.0 + product turns a -0.0 into +0.0 exactly as the add would).  A
// non-finite sum keeps the old value (zero with store) and raises the flag.
template <class Policy>
__device__ __forceinline__ float retained_flux(float old, const FusedParams& P, double flux64, float flux32,
                                               unsigned& flags, bool store)
{
    float st;
    if constexpr (Policy::exact_pow) st = (float)((store ? 0.0 : (double)old) + P.weight * flux64);
    else st = __fmaf_rn(P.weight_f, flux32, store ? 0.0f : old);
    if (isfinite(st)) return st;
    flags |= kStatusNonfiniteMassFlux;
    return store ? 0.0f : old;
}

// The old-state neighbourhood one cell's continuity reads: density at the
// cell and its six face neighbours, the velocities on the cell's upper and
// lower faces, theta, and the stored retained-flux sums.  Neighbours outside
// the grid hold the cell's own value (they are never used).
struct ContinuityStencil
{
    float rho_c, rxp, rxm, ryp, rym, rzp, rzm;
    float uc, uxm, vc, vym, wc, wzm;
    float th;
    float mx, my, mz;
};

// The parts of one cell's continuity.  Every way of loading the stencil (one
// thread per cell, four cells per thread, or marching along i) goes through
// these, so the arithmetic is one sequence.

// Retained flux of the upper x- or y-face: density at the cell and beyond the
// face, the face's velocity, the frame's.
template <class Policy>
__device__ __forceinline__ float retained_lateral(const FusedParams& P, float old, float rc, float rp, float vel,
                                                  double frame, float frame_f, unsigned& flags, bool store)
{
    if constexpr (Policy::exact_pow)
        return retained_flux<Policy>(old, P, 0.5 * ((double)rc + (double)rp) * ((double)vel - frame), 0.0f, flags,
                                     store);
    else
        return retained_flux<Policy>(old, P, 0.0, 0.5f * (rc + rp) * (vel - frame_f), flags, store);
}

// Retained flux of the upper z-face (the lid's own under an open top, else 0).
template <class Policy>
__device__ __forceinline__ float retained_vertical(const FusedParams& P, float old, float rc, float rp, float wc,
                                                   bool zhi, unsigned& flags, bool store)
{
    if constexpr (Policy::exact_pow)
    {
        const double r = (double)rc;
        const double zf = !zhi ? (P.top_open ? r * (double)wc : 0.0) : 0.5 * (r + (double)rp) * (double)wc;
        return retained_flux<Policy>(old, P, zf, 0.0f, flags, store);
    }
    else
    {
        const float zf = !zhi ? (P.top_open ? rc * wc : 0.0f) : 0.5f * (rc + rp) * wc;
        return retained_flux<Policy>(old, P, 0.0, zf, flags, store);
    }
}

// Mass leaving through the upper face less mass entering through the lower.
template <class real>
__device__ __forceinline__ real flux_difference(float rc, float rp, float rm, float vp, float vm)
{
    const real half = (real)0.5;
    const real r = (real)rc;
    const real pos = half * (r + (real)rp) * (real)vp;
    const real neg = half * ((real)rm + r) * (real)vm;
    return pos - neg;
}

template <class real>
__device__ __forceinline__ real flux_difference_z(float rc, float rp, float rm, float wp, float wm, bool zlo, bool zhi)
{
    const real half = (real)0.5;
    const real r = (real)rc;
    const real pos = zhi ? half * (r + (real)rp) * (real)wp : r * (real)wp;
    const real neg = zlo ? half * ((real)rm + r) * (real)wm : (real)0;
    return pos - neg;
}

// The stored continuity tendency from the three differences.
template <class Policy>
__device__ __forceinline__ float continuity_tendency(const FusedParams& P, typename Policy::real dx,
                                                     typename Policy::real dy, typename Policy::real dz)
{
    if constexpr (Policy::exact_pow) return (float)finite_or_zero(-(dx * P.inv_dx + dy * P.inv_dy + dz * P.inv_dz));
    else
    {
        const float drho = -(dx * P.inv_dx_f + dy * P.inv_dy_f + dz * P.inv_dz_f);
        return isfinite(drho) ? drho : 0.0f;
    }
}

// What one cell's continuity forms: the stored tendency, the new density and
// pressure and the retained fluxes of its three upper faces (meaningful where
// the face exists: i < nx-1, j < ny-1, every k).
struct ContinuityResult
{
    float drho, rho, p;
    float mx, my, mz;
};

// Continuity, rho forward Euler and EOS of cell (i, j, k) from its loaded
// stencil; with flux the retained fluxes are written (store_flux) or
// accumulated.
template <class Policy>
__device__ __forceinline__ ContinuityResult continuity_eos_point(const FusedParams& P, const ContinuityStencil& s,
                                                                 bool xlo, bool xhi, bool ylo, bool yhi, int k,
                                                                 const double* __restrict__ rho0,
                                                                 const float4* __restrict__ eos0, bool flux,
                                                                 unsigned& flags, bool store_flux)
{
    using real = typename Policy::real;
    const bool zlo = k > 0, zhi = k + 1 < P.d.nz;
    ContinuityResult o;
    o.mx = s.mx;
    o.my = s.my;
    o.mz = s.mz;
    if (flux)
    {
        if (xhi)
            o.mx = retained_lateral<Policy>(P, s.mx, s.rho_c, s.rxp, s.uc, P.frame_u, P.frame_u_f, flags, store_flux);
        if (yhi)
            o.my = retained_lateral<Policy>(P, s.my, s.rho_c, s.ryp, s.vc, P.frame_v, P.frame_v_f, flags, store_flux);
        o.mz = retained_vertical<Policy>(P, s.mz, s.rho_c, s.rzp, s.wc, zhi, flags, store_flux);
    }
    o.drho = 0.0f;
    if (xlo && xhi && ylo && yhi)
        o.drho = continuity_tendency<Policy>(P, flux_difference<real>(s.rho_c, s.rxp, s.rxm, s.uc, s.uxm),
                                             flux_difference<real>(s.rho_c, s.ryp, s.rym, s.vc, s.vym),
                                             flux_difference_z<real>(s.rho_c, s.rzp, s.rzm, s.wc, s.wzm, zlo, zhi));
    o.rho = substep_density<Policy>(P, s.rho_c, o.drho, rho0, k);
    o.p = substep_pressure<Policy>(P, eos0, k, o.rho, s.th);
    return o;
}

// continuity_eos_point of cell c = (i, j, k), stored.
template <class Policy>
__device__ __forceinline__ void continuity_eos_values(const FusedParams& P, const ContinuityStencil& s, int i, int j,
                                                      int k, int c, const double* __restrict__ rho0,
                                                      const float4* __restrict__ eos0, float* __restrict__ rho_out,
                                                      float* __restrict__ p_out, float* __restrict__ drho_out,
                                                      float* __restrict__ mfx, float* __restrict__ mfy,
                                                      float* __restrict__ mfz, unsigned& flags, bool store_flux,
                                                      float* __restrict__ rho_copy)
{
    const Dims d = P.d;
    const bool xhi = i < d.nx - 1, yhi = j < d.ny - 1;
    const bool flux = mfx != nullptr;
    if (rho_copy != nullptr) rho_copy[c] = s.rho_c;
    const ContinuityResult o =
        continuity_eos_point<Policy>(P, s, i >= 1, xhi, j >= 1, yhi, k, rho0, eos0, flux, flags, store_flux);
    if (flux)
    {
        if (xhi) mfx[c] = o.mx;
        if (yhi) mfy[c] = o.my;
        mfz[c] = o.mz;
    }
    if (drho_out != nullptr) drho_out[c] = o.drho;
    rho_out[c] = o.rho;
    p_out[c] = o.p;
}

// Loads cell c = (i, j, k)'s continuity stencil (acc: the stored retained-flux
// sums too).  Neighbours outside the grid read the cell itself.
__device__ __forceinline__ ContinuityStencil continuity_load(const Dims& d, const float* __restrict__ rho,
                                                             const float* __restrict__ u,
                                                             const float* __restrict__ v,
                                                             const float* __restrict__ w,
                                                             const float* __restrict__ theta, const float* mfx,
                                                             const float* mfy, const float* mfz, bool acc, int c,
                                                             int i, int j, int k)
{
    const int sx = d.sx(), sy = d.sy();
    const bool xlo = i >= 1, xhi = i < d.nx - 1, ylo = j >= 1, yhi = j < d.ny - 1;
    const bool zlo = k > 0, zhi = k + 1 < d.nz;
    ContinuityStencil s;
    s.rho_c = rho[c];
    s.rxp = rho[xhi ? c + sx : c];
    s.rxm = rho[xlo ? c - sx : c];
    s.ryp = rho[yhi ? c + sy : c];
    s.rym = rho[ylo ? c - sy : c];
    s.rzp = rho[zhi ? c + 1 : c];
    s.rzm = rho[zlo ? c - 1 : c];
    s.uc = u[c];
    s.uxm = u[xlo ? c - sx : c];
    s.vc = v[c];
    s.vym = v[ylo ? c - sy : c];
    s.wc = w[c];
    s.wzm = w[zlo ? c - 1 : c];
    s.th = theta[c];
    s.mx = acc ? mfx[c] : 0.0f;
    s.my = acc ? mfy[c] : 0.0f;
    s.mz = acc ? mfz[c] : 0.0f;
    return s;
}

// Continuity, rho forward Euler and EOS for cell c.  With store_flux the
// retained fluxes are written rather than accumulated and rho_copy (when
// given) receives the pre-substep density (the transport context's
// beginning density).  Every load is issued before any arithmetic (indices of
// neighbours outside the grid are clamped to the cell; those values are not
// used), so a thread has all of its memory requests in flight at once.
template <class Policy>
__device__ __forceinline__ void continuity_eos_cell(const FusedParams& P, const float* __restrict__ rho,
                                                    const float* __restrict__ u, const float* __restrict__ v,
                                                    const float* __restrict__ w, const float* __restrict__ theta,
                                                    const double* __restrict__ rho0,
                                                    const float4* __restrict__ eos0, float* __restrict__ rho_out,
                                                    float* __restrict__ p_out, float* __restrict__ drho_out,
                                                    float* __restrict__ mfx, float* __restrict__ mfy,
                                                    float* __restrict__ mfz, int c, unsigned& flags, bool store_flux,
                                                    float* __restrict__ rho_copy)
{
    int i, j, k;
    decompose(P.d, c, i, j, k);
    if (k >= P.d.nz) return;
    const ContinuityStencil s =
        continuity_load(P.d, rho, u, v, w, theta, mfx, mfy, mfz, mfx != nullptr && !store_flux, c, i, j, k);
    continuity_eos_values<Policy>(P, s, i, j, k, c, rho0, eos0, rho_out, p_out, drho_out, mfx, mfy, mfz, flags,
                                  store_flux, rho_copy);
}

// The same continuity for the cells (i0 .. i1-1, j, k) of one grid row along
// x, marching in i: the density of planes i-1, i and the x-velocity of plane
// i-1 carry over in registers from the previous cell, so a cell loads one new
// x-neighbour instead of three, and its neighbour offsets and boundary flags
// in j and k are formed once per row.  q = j pz + k.
template <class Policy>
__device__ __forceinline__ void continuity_eos_march(const FusedParams& P, const float* __restrict__ rho,
                                                     const float* __restrict__ u, const float* __restrict__ v,
                                                     const float* __restrict__ w, const float* __restrict__ theta,
                                                     const double* __restrict__ rho0,
                                                     const float4* __restrict__ eos0, float* __restrict__ rho_out,
                                                     float* __restrict__ p_out, float* __restrict__ mfx,
                                                     float* __restrict__ mfy, float* __restrict__ mfz, int i0, int i1,
                                                     int j, int k, int q, unsigned& flags, bool store_flux,
                                                     float* __restrict__ rho_copy)
{
    const Dims d = P.d;
    const int sx = d.sx();
    const int oyp = j < d.ny - 1 ? d.sy() : 0, oym = j >= 1 ? -d.sy() : 0;
    const int ozp = k + 1 < d.nz ? 1 : 0, ozm = k > 0 ? -1 : 0;
    const bool acc = mfx != nullptr && !store_flux;
    int c = i0 * sx + q;
    float r_m = rho[i0 >= 1 ? c - sx : c];
    float r_c = rho[c];
    float u_m = u[i0 >= 1 ? c - sx : c];
    for (int i = i0; i < i1; ++i, c += sx)
    {
        ContinuityStencil s;
        s.rho_c = r_c;
        s.rxm = r_m;
        s.rxp = rho[i < d.nx - 1 ? c + sx : c];
        s.ryp = rho[c + oyp];
        s.rym = rho[c + oym];
        s.rzp = rho[c + ozp];
        s.rzm = rho[c + ozm];
        s.uc = u[c];
        s.uxm = u_m;
        s.vc = v[c];
        s.vym = v[c + oym];
        s.wc = w[c];
        s.wzm = w[c + ozm];
        s.th = theta[c];
        s.mx = acc ? mfx[c] : 0.0f;
        s.my = acc ? mfy[c] : 0.0f;
        s.mz = acc ? mfz[c] : 0.0f;
        continuity_eos_values<Policy>(P, s, i, j, k, c, rho0, eos0, rho_out, p_out, nullptr, mfx, mfy, mfz, flags,
                                      store_flux, rho_copy);
        r_m = r_c;
        r_c = s.rxp;
        u_m = s.uc;
    }
}

template <class Policy>
static __global__ void __launch_bounds__(256) split_continuity_eos_kernel(
    FusedParams P, const float* __restrict__ rho, const float* __restrict__ u, const float* __restrict__ v,
    const float* __restrict__ w, const float* __restrict__ theta, const double* __restrict__ rho0,
    const float4* __restrict__ eos0, float* __restrict__ rho_out, float* __restrict__ p_out,
    float* __restrict__ drho_out, float* __restrict__ mfx, float* __restrict__ mfy, float* __restrict__ mfz,
    unsigned* __restrict__ status)
{
    grid_dependency();
    const int n = P.d.cells();
    unsigned flags = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
        continuity_eos_cell<Policy>(P, rho, u, v, w, theta, rho0, eos0, rho_out, p_out, drho_out, mfx, mfy, mfz, c,
                                    flags, false, nullptr);
    if (flags) atomicOr(status, flags);
}

// Momentum forward Euler for the faces of cell c.  Face c reads only its own
// old velocity, so u_out may alias u (in-place update).
// Stores the new face velocities of cell c, with the vertical closure of its
// column when fuse_vertical asks for it (see momentum_cell).  (Handing the
// top values to the cell above through a warp shuffle, so that every lane
// stores its own cell, measured slower than these scattered stores.)
__device__ __forceinline__ void momentum_store(const Dims& d, int i, int j, int k, int c, int fuse_vertical, float un,
                                               float vn, float wn, float* u_out, float* v_out, float* w_out)
{
    if ((fuse_vertical & 1) && bc_inner_column(d, i, j))
    {
        if (k == d.nz - 1) return;  // written by the cell below
        if (k == 0 && (fuse_vertical & 2))
        {
            un = 0.0f;
            vn = 0.0f;
        }
        if (k == d.nz - 2)
        {
            u_out[c + 1] = un;
            v_out[c + 1] = vn;
            w_out[c + 1] = (fuse_vertical & 4) ? wn : 0.0f;
        }
    }
    u_out[c] = un;
    v_out[c] = vn;
    w_out[c] = wn;
}

// fuse_vertical (kFuse* bits): the momentum pass also applies the vertical
// closure (bc_vertical_column) to the columns no lateral closure writes or
// reads (bc_inner_column): the no-slip bottom zeros u and v at k = 0, the cell
// at k = nz-2 writes its new u, v and w (or 0 under a rigid top) into level
// nz-1 as well, and the cell at nz-1 does not store.
enum : int
{
    kFuseVertical = 1,
    kFuseNoSlipBottom = 2,
    kFuseOpenTop = 4
};

// The new-state neighbourhood of one cell's momentum: density and pressure at
// the cell and its upper x, y and z neighbours, and the cell's old face
// velocities.
struct MomentumStencil
{
    float rc, rx, ry, rz;
    float pc, px, py, pz;
    float uc, vc, wc;
};

// The new face velocities of cell (i, j, k) from its loaded stencil (interior:
// 1 <= i < nx-1, 1 <= j < ny-1, k < nz-1; elsewhere only the clamp acts).
template <class Policy>
__device__ __forceinline__ float3 momentum_point(const FusedParams& P, const MomentumStencil& s, bool interior, int k,
                                                 const double* __restrict__ p0,
                                                 const float2* __restrict__ dp0_split)
{
    using real = typename Policy::real;
    float du = 0.0f, dv = 0.0f, dw = 0.0f;
    if constexpr (sizeof(real) == 8)
    {
        if (interior)
        {
            const double rcd = (double)s.rc;
            const double rho_x = 0.5 * (rcd + (double)s.rx);
            const double rho_y = 0.5 * (rcd + (double)s.ry);
            const double rho_z = 0.5 * (rcd + (double)s.rz);
            const double pcd = (double)s.pc;
            const double dp0_dz = (p0[k + 1] - p0[k]) * P.inv_dz;
            du = (float)finite_or_zero(-((double)s.px - pcd) * P.inv_dx / safe_rho(rho_x));
            dv = (float)finite_or_zero(-((double)s.py - pcd) * P.inv_dy / safe_rho(rho_y));
            dw = (float)finite_or_zero(-((((double)s.pz - pcd) * P.inv_dz) - dp0_dz) / safe_rho(rho_z));
        }
        return make_float3(clamp_value((float)((double)s.uc + (double)du * P.dt_small), 0.0f, -P.wind_h, P.wind_h),
                           clamp_value((float)((double)s.vc + (double)dv * P.dt_small), 0.0f, -P.wind_h, P.wind_h),
                           clamp_value((float)((double)s.wc + (double)dw * P.dt_small), 0.0f, -P.wind_v, P.wind_v));
    }
    else
    {
        if (interior)
        {
            const float2 dp0 = dp0_split[k];
            const float rho_x = 0.5f * (s.rc + s.rx);
            const float rho_y = 0.5f * (s.rc + s.ry);
            const float rho_z = 0.5f * (s.rc + s.rz);
            const float dpz = ((s.pz - s.pc) - dp0.x) - dp0.y;
            const float sxr = (isfinite(rho_x) && rho_x > 1.0e-6f) ? rho_x : 1.0f;
            const float syr = (isfinite(rho_y) && rho_y > 1.0e-6f) ? rho_y : 1.0f;
            const float szr = (isfinite(rho_z) && rho_z > 1.0e-6f) ? rho_z : 1.0f;
            const float a = -(s.px - s.pc) * P.inv_dx_f * rcp_normal(sxr);  // the densities exceed 1e-6
            const float b = -(s.py - s.pc) * P.inv_dy_f * rcp_normal(syr);
            const float cz = -dpz * P.inv_dz_f * rcp_normal(szr);
            du = isfinite(a) ? a : 0.0f;
            dv = isfinite(b) ? b : 0.0f;
            dw = isfinite(cz) ? cz : 0.0f;
        }
        const float dt = P.dt_f;
        return make_float3(clamp_value(__fmaf_rn(du, dt, s.uc), 0.0f, -P.wind_h, P.wind_h),
                           clamp_value(__fmaf_rn(dv, dt, s.vc), 0.0f, -P.wind_h, P.wind_h),
                           clamp_value(__fmaf_rn(dw, dt, s.wc), 0.0f, -P.wind_v, P.wind_v));
    }
}

// momentum_point of cell c = (i, j, k), stored (see momentum_store).
template <class Policy>
__device__ __forceinline__ void momentum_values(const FusedParams& P, const MomentumStencil& s, int i, int j, int k,
                                                int c, const double* __restrict__ p0,
                                                const float2* __restrict__ dp0_split, float* u_out, float* v_out,
                                                float* w_out, int fuse_vertical)
{
    const Dims d = P.d;
    const bool interior = i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1 && k < d.nz - 1;
    const float3 n = momentum_point<Policy>(P, s, interior, k, p0, dp0_split);
    momentum_store(d, i, j, k, c, fuse_vertical, n.x, n.y, n.z, u_out, v_out, w_out);
}

// Loads cell c = (i, j, k)'s momentum stencil; outside the interior the
// neighbour indices fall back to the cell itself (those values are not used).
__device__ __forceinline__ MomentumStencil momentum_load(const Dims& d, const float* __restrict__ rho,
                                                         const float* __restrict__ p, const float* u, const float* v,
                                                         const float* w, int c, int i, int j, int k)
{
    const bool interior = i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1 && k < d.nz - 1;
    const int cx = interior ? c + d.sx() : c, cy = interior ? c + d.sy() : c, cz1 = interior ? c + 1 : c;
    MomentumStencil s;
    s.rc = rho[c];
    s.rx = rho[cx];
    s.ry = rho[cy];
    s.rz = rho[cz1];
    s.pc = p[c];
    s.px = p[cx];
    s.py = p[cy];
    s.pz = p[cz1];
    s.uc = u[c];
    s.vc = v[c];
    s.wc = w[c];
    return s;
}

template <class Policy>
__device__ __forceinline__ void momentum_cell(const FusedParams& P, const float* __restrict__ rho,
                                              const float* __restrict__ p, const double* __restrict__ p0,
                                              const float2* __restrict__ dp0_split, const float* u, const float* v,
                                              const float* w, float* u_out, float* v_out, float* w_out, int c,
                                              int fuse_vertical = 0)
{
    int i, j, k;
    decompose(P.d, c, i, j, k);
    if (k >= P.d.nz) return;
    const MomentumStencil s = momentum_load(P.d, rho, p, u, v, w, c, i, j, k);
    momentum_values<Policy>(P, s, i, j, k, c, p0, dp0_split, u_out, v_out, w_out, fuse_vertical);
}

// The same momentum for the cells (i0 .. i1-1, j, k) of one row along x,
// marching in i: the new density and pressure of plane i+1 loaded for cell i
// are those of cell i+1, so they carry over in registers.  q = j pz + k.
template <class Policy>
__device__ __forceinline__ void momentum_march(const FusedParams& P, const float* __restrict__ rho,
                                               const float* __restrict__ p, const double* __restrict__ p0,
                                               const float2* __restrict__ dp0_split, float* u, float* v, float* w,
                                               int i0, int i1, int j, int k, int q, int fuse_vertical)
{
    const Dims d = P.d;
    const int sx = d.sx();
    const int oy = j < d.ny - 1 ? d.sy() : 0, oz = k < d.nz - 1 ? 1 : 0;
    int c = i0 * sx + q;
    float rc = rho[c], pc = p[c];
    for (int i = i0; i < i1; ++i, c += sx)
    {
        MomentumStencil s;
        const int cx = i < d.nx - 1 ? c + sx : c;
        s.rc = rc;
        s.pc = pc;
        s.rx = rho[cx];
        s.px = p[cx];
        s.ry = rho[c + oy];
        s.py = p[c + oy];
        s.rz = rho[c + oz];
        s.pz = p[c + oz];
        s.uc = u[c];
        s.vc = v[c];
        s.wc = w[c];
        momentum_values<Policy>(P, s, i, j, k, c, p0, dp0_split, u, v, w, fuse_vertical);
        rc = s.rx;
        pc = s.px;
    }
}

// ---- Four vertically adjacent cells per thread -----------------------------
// Cells c .. c + 3 with k a multiple of 4, of a grid whose columns start on
// 16-byte boundaries: they lie in one column, share i and j, and each field's
// values at the four cells and at the four shifted by +-sx or +-sy are one
// aligned 16-byte load.  The cell passes' limit is the issue of instructions
// (291 and 144 a cell in the one-cell and marching forms, two thirds of the
// slots used), most of them loads, addresses, index arithmetic and range
// tests, which the four cells share here.  Each cell's arithmetic is the
// one-cell form's.
struct Quad
{
    float v[4];
};

// Keeps the compiler from moving loads across it (no instruction).
__device__ __forceinline__ void load_stage() { asm volatile("" ::: "memory"); }

__device__ __forceinline__ Quad load_quad(const float* __restrict__ f, int c)
{
    const float4 t = *reinterpret_cast<const float4*>(f + c);
    return Quad{{t.x, t.y, t.z, t.w}};
}

__device__ __forceinline__ void store_quad(float* f, int c, const Quad& q)
{
    *reinterpret_cast<float4*>(f + c) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}

template <class Policy>
__device__ __forceinline__ void continuity_eos_quad(const FusedParams& P, const float* __restrict__ rho,
                                                    const float* __restrict__ u, const float* __restrict__ v,
                                                    const float* __restrict__ w, const float* __restrict__ theta,
                                                    const double* __restrict__ rho0,
                                                    const float4* __restrict__ eos0, float* __restrict__ rho_out,
                                                    float* __restrict__ p_out, float* __restrict__ mfx,
                                                    float* __restrict__ mfy, float* __restrict__ mfz, int c,
                                                    unsigned& flags, bool store_flux, float* __restrict__ rho_copy)
{
    const Dims d = P.d;
    int i, j, k;
    decompose(d, c, i, j, k);
    const int sx = d.sx(), sy = d.sy();
    const bool xlo = i >= 1, xhi = i < d.nx - 1, ylo = j >= 1, yhi = j < d.ny - 1;
    using real = typename Policy::real;
    const bool flux = mfx != nullptr, acc = flux && !store_flux;
    const bool interior = xlo && xhi && ylo && yhi;
    // Axis by axis: each axis' loads end at a barrier to the compiler's
    // reordering, so that the registers of one serve the next and the kernel
    // runs at eight CTAs of 128 threads an SM instead of four or five.
    unsigned bad[4] = {0, 0, 0, 0};
    const Quad r = load_quad(rho, c);
    if (rho_copy != nullptr) store_quad(rho_copy, c, r);
    real dx[4], dy[4], dz[4];
    {
        const Quad rp = load_quad(rho, xhi ? c + sx : c), rm = load_quad(rho, xlo ? c - sx : c);
        const Quad vp = load_quad(u, c), vm = load_quad(u, xlo ? c - sx : c);
        Quad m{};
        if (acc) m = load_quad(mfx, c);
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            if (flux && xhi)
                m.v[q] = retained_lateral<Policy>(P, m.v[q], r.v[q], rp.v[q], vp.v[q], P.frame_u, P.frame_u_f, bad[q],
                                                  store_flux);
            dx[q] = flux_difference<real>(r.v[q], rp.v[q], rm.v[q], vp.v[q], vm.v[q]);
        }
        if (flux && xhi) store_quad(mfx, c, m);
    }
    load_stage();
    {
        const Quad rp = load_quad(rho, yhi ? c + sy : c), rm = load_quad(rho, ylo ? c - sy : c);
        const Quad vp = load_quad(v, c), vm = load_quad(v, ylo ? c - sy : c);
        Quad m{};
        if (acc) m = load_quad(mfy, c);
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            if (flux && yhi)
                m.v[q] = retained_lateral<Policy>(P, m.v[q], r.v[q], rp.v[q], vp.v[q], P.frame_v, P.frame_v_f, bad[q],
                                                  store_flux);
            dy[q] = flux_difference<real>(r.v[q], rp.v[q], rm.v[q], vp.v[q], vm.v[q]);
        }
        if (flux && yhi) store_quad(mfy, c, m);
    }
    load_stage();
    const Quad th = load_quad(theta, c);
    {
        const float rzm = rho[k > 0 ? c - 1 : c], rzp = rho[k + 4 < d.nz ? c + 4 : c + 3];
        const Quad wc = load_quad(w, c);
        const float wzm = w[k > 0 ? c - 1 : c];
        Quad m{};
        if (acc) m = load_quad(mfz, c);
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            const float rp = q < 3 ? r.v[q < 3 ? q + 1 : 3] : rzp, rm = q > 0 ? r.v[q > 0 ? q - 1 : 0] : rzm;
            const float wm = q > 0 ? wc.v[q > 0 ? q - 1 : 0] : wzm;
            const bool zlo = k + q > 0, zhi = k + q + 1 < d.nz;
            if (flux)
                m.v[q] = retained_vertical<Policy>(P, m.v[q], r.v[q], rp, wc.v[q], zhi, bad[q], store_flux);
            dz[q] = flux_difference_z<real>(r.v[q], rp, rm, wc.v[q], wm, zlo, zhi);
        }
        if (flux) store_quad(mfz, c, m);
    }
    Quad rn, pn;
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        const float drho = interior ? continuity_tendency<Policy>(P, dx[q], dy[q], dz[q]) : 0.0f;
        rn.v[q] = substep_density<Policy>(P, r.v[q], drho, rho0, k + q);
        pn.v[q] = substep_pressure<Policy>(P, eos0, k + q, rn.v[q], th.v[q]);
        if (k + q < d.nz) flags |= bad[q];  // a padded cell's values are not state
    }
    store_quad(rho_out, c, rn);
    store_quad(p_out, c, pn);
}

template <class Policy>
__device__ __forceinline__ void momentum_quad(const FusedParams& P, const float* __restrict__ rho,
                                              const float* __restrict__ p, const double* __restrict__ p0,
                                              const float2* __restrict__ dp0_split, const float* u, const float* v,
                                              const float* w, float* u_out, float* v_out, float* w_out, int c,
                                              int fuse_vertical)
{
    const Dims d = P.d;
    int i, j, k;
    decompose(d, c, i, j, k);
    const bool ij = i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1;
    const int cx = ij ? c + d.sx() : c, cy = ij ? c + d.sy() : c, cz = k + 4 < d.nz ? c + 4 : c + 3;
    const Quad r = load_quad(rho, c), rx = load_quad(rho, cx), ry = load_quad(rho, cy);
    const Quad pc = load_quad(p, c), px = load_quad(p, cx), py = load_quad(p, cy);
    const float rz = rho[cz], pz = p[cz];
    Quad un = load_quad(u, c), vn = load_quad(v, c), wn = load_quad(w, c);
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        MomentumStencil s;
        s.rc = r.v[q];
        s.rx = rx.v[q];
        s.ry = ry.v[q];
        s.rz = q < 3 ? r.v[q < 3 ? q + 1 : 3] : rz;
        s.pc = pc.v[q];
        s.px = px.v[q];
        s.py = py.v[q];
        s.pz = q < 3 ? pc.v[q < 3 ? q + 1 : 3] : pz;
        s.uc = un.v[q];
        s.vc = vn.v[q];
        s.wc = wn.v[q];
        const float3 n = momentum_point<Policy>(P, s, ij && k + q < d.nz - 1, k + q, p0, dp0_split);
        un.v[q] = n.x;
        vn.v[q] = n.y;
        wn.v[q] = n.z;
    }
    if ((fuse_vertical & kFuseVertical) && bc_inner_column(d, i, j))
    {
        // momentum_store's vertical closure on the four cells; the top level
        // is cell kt of them.
        if (k == 0 && (fuse_vertical & kFuseNoSlipBottom)) un.v[0] = vn.v[0] = 0.0f;
        const int kt = d.nz - 1 - k;
        const bool open = (fuse_vertical & kFuseOpenTop) != 0;
        if (kt == 0) return;  // the level below writes it, and the rest is padding
#pragma unroll
        for (int q = 1; q < 4; ++q)
            if (q == kt)
            {
                un.v[q] = un.v[q - 1];
                vn.v[q] = vn.v[q - 1];
                wn.v[q] = open ? wn.v[q - 1] : 0.0f;
            }
        if (kt == 4)
        {
            u_out[c + 4] = un.v[3];
            v_out[c + 4] = vn.v[3];
            w_out[c + 4] = open ? wn.v[3] : 0.0f;
        }
    }
    store_quad(u_out, c, un);
    store_quad(v_out, c, vn);
    store_quad(w_out, c, wn);
}

constexpr int kQuadBlock = 128;  // threads of a quad kernel

// CTAs per SM that a quad kernel's launch bounds ask for.  FP32 at 8 (64
// registers without spills; 512x512x128, ps per cell, continuity / momentum at
// 8, 7, 6: 8.98 / 4.70, 9.72 / 4.81, 10.27; one cell per thread 11.1 / 6.8),
// reference precision at 7 (72; four steps of 3.0 million cells at 8 / 7 / 6:
// 1.51 / 1.48 / 1.53 and 1.13 / 1.09 / 1.12 ms).
template <class Policy>
constexpr int kQuadCtas = sizeof(typename Policy::real) == 4 ? 8 : 7;

// Cells from which the quad kernels are launched: below, a cell per thread
// fills the SMs better than the quad saves instructions (four CTAs of quads an
// SM on the B200's 148 SMs).  The line lies between those of the two precisions;
// a substep of the per-operation loop, us with quads / one cell per thread:
// FP32 164 thousand cells 14.0 / 13.5, 207 15.1 / 15.5, 310 17.1 / 17.4, 1024
// 25.4 / 30.2; reference precision 207 18.1 / 17.3, 310 21.0 / 20.5, 369
// 20.9 / 20.8, 433 22.8 / 23.6, 1024 32.9 / 38.2.
constexpr long long kQuadCells = 4LL * kQuadBlock * 4 * 148;

template <class Policy>
static __global__ void __launch_bounds__(kQuadBlock, kQuadCtas<Policy>) split_continuity_quad_kernel(
    FusedParams P, const float* __restrict__ rho, const float* __restrict__ u, const float* __restrict__ v,
    const float* __restrict__ w, const float* __restrict__ theta, const double* __restrict__ rho0,
    const float4* __restrict__ eos0, float* __restrict__ rho_out, float* __restrict__ p_out,
    float* __restrict__ mfx, float* __restrict__ mfy, float* __restrict__ mfz, unsigned* __restrict__ status)
{
    grid_dependency();
    const int n = P.d.cells();
    unsigned flags = 0;
    for (int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x); c < n; c += 4 * gridDim.x * blockDim.x)
        continuity_eos_quad<Policy>(P, rho, u, v, w, theta, rho0, eos0, rho_out, p_out, mfx, mfy, mfz, c, flags, false,
                                    nullptr);
    if (flags) atomicOr(status, flags);
}

template <class Policy>
static __global__ void __launch_bounds__(kQuadBlock, kQuadCtas<Policy>) split_momentum_quad_kernel(
    FusedParams P, const float* __restrict__ rho, const float* __restrict__ p, const double* __restrict__ p0,
    const float2* __restrict__ dp0_split, const float* __restrict__ u, const float* __restrict__ v,
    const float* __restrict__ w, float* __restrict__ u_out, float* __restrict__ v_out, float* __restrict__ w_out,
    int fuse_vertical)
{
    grid_dependency();
    const int n = P.d.cells();
    for (int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x); c < n; c += 4 * gridDim.x * blockDim.x)
        momentum_quad<Policy>(P, rho, p, p0, dp0_split, u, v, w, u_out, v_out, w_out, c, fuse_vertical);
}

template <class Policy>
static __global__ void __launch_bounds__(256) split_momentum_kernel(
    FusedParams P, const float* __restrict__ rho, const float* __restrict__ p, const double* __restrict__ p0,
    const float2* __restrict__ dp0_split, const float* __restrict__ u, const float* __restrict__ v,
    const float* __restrict__ w, float* __restrict__ u_out, float* __restrict__ v_out, float* __restrict__ w_out,
    int fuse_vertical)
{
    grid_dependency();
    const int n = P.d.cells();
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
        momentum_cell<Policy>(P, rho, p, p0, dp0_split, u, v, w, u_out, v_out, w_out, c, fuse_vertical);
}

}  // namespace nimbus
