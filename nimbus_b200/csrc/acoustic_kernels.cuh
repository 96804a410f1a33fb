// Acoustic substep kernels of the Klemp-Wilhelmson split-explicit loop on
// the flat Cartesian C-grid, reference-precision form: FP32 storage, FP64
// interior arithmetic in the reference's own operation order.  This file is
// compiled with --fmad=false so no multiply-add is contracted, which keeps
// every stored value identical to the reference CPU solver's.
//
// One substep is two full-grid passes plus the boundary pass:
//   continuity_eos : retained mass-flux accumulation from the pre-substep
//                    state, continuity tendency, rho forward Euler + clamp,
//                    EOS pressure + clamp.  rho is written to the other half
//                    of a ping-pong pair (neighbours still need the old rho);
//                    p is written in place (the old p is never read).
//   momentum       : u,v,w forward Euler from the new pressure gradient.
//   bc_ring        : the boundary closure in the reference's face order
//                    W,E -> S,N -> vertical, one launch (bc_ring_levels).
#pragma once

#include "power_table.cuh"
#include "stencil_common.cuh"

namespace nimbus
{

struct AcousticParams
{
    Dims d;
    double inv_dx, inv_dy, inv_dz;
    double dt_small;
    double gamma;
    float rho_min, rho_max, p_min, p_max, p_ref_fallback, wind_h, wind_v;
    // Retained mass flux (accumulated when mfx != nullptr).
    double weight;
    double frame_u, frame_v;
    int top_open;
};

// Pass 1+2 of acoustic_cgrid_fast.cpp:47-157 and the Host-precision flux
// accumulation of advection_cartesian.cpp:743-849 (cartesian_mass_flux.hpp:57-75,381-393).
static __global__ void __launch_bounds__(256) acoustic_continuity_eos_kernel(
    AcousticParams P, const float* __restrict__ rho, const float* __restrict__ u, const float* __restrict__ v,
    const float* __restrict__ w, const float* __restrict__ theta, const double* __restrict__ rho0,
    float* __restrict__ rho_out, float* __restrict__ p_out, float* __restrict__ drho_out,
    float* __restrict__ mfx, float* __restrict__ mfy, float* __restrict__ mfz, unsigned* __restrict__ status)
{
    const Dims d = P.d;
    const int n = d.cells();
    const int sx = d.sx(), sy = d.sy();
    unsigned flags = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    {
        int i, j, k;
        decompose(d, c, i, j, k);
        const double rc = (double)rho[c];

        if (mfx != nullptr)
        {
            const double weight = P.weight;
            if (i < d.nx - 1)
            {
                const double vel = (double)u[c] - P.frame_u;
                const double flux = 0.5 * (rc + (double)rho[c + sx]) * vel;
                const double next = (double)mfx[c] + weight * flux;
                const float stored = (float)next;
                if (isfinite(next) && isfinite(stored)) mfx[c] = stored;
                else flags |= kStatusNonfiniteMassFlux;
            }
            if (j < d.ny - 1)
            {
                const double vel = (double)v[c] - P.frame_v;
                const double flux = 0.5 * (rc + (double)rho[c + sy]) * vel;
                const double next = (double)mfy[c] + weight * flux;
                const float stored = (float)next;
                if (isfinite(next) && isfinite(stored)) mfy[c] = stored;
                else flags |= kStatusNonfiniteMassFlux;
            }
            double zflux;
            if (k == d.nz - 1) zflux = P.top_open ? rc * (double)w[c] : 0.0;
            else zflux = 0.5 * (rc + (double)rho[c + 1]) * (double)w[c];
            const double znext = (double)mfz[c] + weight * zflux;
            const float zstored = (float)znext;
            if (isfinite(znext) && isfinite(zstored)) mfz[c] = zstored;
            else flags |= kStatusNonfiniteMassFlux;
        }

        double drho = 0.0;
        if (i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1)
        {
            const double fx_pos = 0.5 * (rc + (double)rho[c + sx]) * (double)u[c];
            const double fx_neg = 0.5 * ((double)rho[c - sx] + rc) * (double)u[c - sx];
            const double fy_pos = 0.5 * (rc + (double)rho[c + sy]) * (double)v[c];
            const double fy_neg = 0.5 * ((double)rho[c - sy] + rc) * (double)v[c - sy];
            const double fz_pos = (k + 1 < d.nz) ? 0.5 * (rc + (double)rho[c + 1]) * (double)w[c] : rc * (double)w[c];
            const double fz_neg = (k > 0) ? 0.5 * ((double)rho[c - 1] + rc) * (double)w[c - 1] : 0.0;
            drho = -((fx_pos - fx_neg) * P.inv_dx + (fy_pos - fy_neg) * P.inv_dy + (fz_pos - fz_neg) * P.inv_dz);
        }
        const float drho_stored = (float)finite_or_zero(drho);
        if (drho_out != nullptr) drho_out[c] = drho_stored;

        double rho_new = rc + (double)drho_stored * P.dt_small;
        if (!isfinite(rho_new) || rho_new <= 0.0)
        {
            const double base = rho0[k];
            rho_new = (0.1 < base) ? base : 0.1;
        }
        const float rho_stored = clamp_value((float)rho_new, 1.0f, P.rho_min, P.rho_max);
        rho_out[c] = rho_stored;

        double p_new = (double)P.p_ref_fallback;
        const double th = (double)theta[c];
        if (th > 0.0) p_new = kP00 * eos_power((double)rho_stored * kRd * th / kP00, P.gamma);
        if (!isfinite(p_new) || p_new <= 0.0) p_new = (double)P.p_ref_fallback;
        p_out[c] = clamp_value((float)p_new, 101325.0f, P.p_min, P.p_max);
    }
    if (flags) atomicOr(status, flags);
}

// Pass 3 of acoustic_cgrid_fast.cpp:159-215, in place on u,v,w.
static __global__ void __launch_bounds__(256) acoustic_momentum_kernel(
    AcousticParams P, const float* __restrict__ rho, const float* __restrict__ p, const double* __restrict__ p0,
    float* __restrict__ u, float* __restrict__ v, float* __restrict__ w)
{
    const Dims d = P.d;
    const int n = d.cells();
    const int sx = d.sx(), sy = d.sy();
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    {
        int i, j, k;
        decompose(d, c, i, j, k);
        float du = 0.0f, dv = 0.0f, dw = 0.0f;
        if (i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1 && k < d.nz - 1)
        {
            const double rc = (double)rho[c];
            const double rho_x = 0.5 * (rc + (double)rho[c + sx]);
            const double rho_y = 0.5 * (rc + (double)rho[c + sy]);
            const double rho_z = 0.5 * (rc + (double)rho[c + 1]);
            const double dp0_dz = (p0[k + 1] - p0[k]) * P.inv_dz;
            const double pc = (double)p[c];
            du = (float)finite_or_zero(-((double)p[c + sx] - pc) * P.inv_dx / safe_rho(rho_x));
            dv = (float)finite_or_zero(-((double)p[c + sy] - pc) * P.inv_dy / safe_rho(rho_y));
            dw = (float)finite_or_zero(-((((double)p[c + 1] - pc) * P.inv_dz) - dp0_dz) / safe_rho(rho_z));
        }
        u[c] = clamp_value((float)((double)u[c] + (double)du * P.dt_small), 0.0f, -P.wind_h, P.wind_h);
        v[c] = clamp_value((float)((double)v[c] + (double)dv * P.dt_small), 0.0f, -P.wind_h, P.wind_h);
        w[c] = clamp_value((float)((double)w[c] + (double)dw * P.dt_small), 0.0f, -P.wind_v, P.wind_v);
    }
}

struct BoundaryParams
{
    Dims d;
    int west, east, south, north, bottom, top;
    float dt_rad;     // (float)dt_small; 0 = refresh only
    float inv_dx, inv_dy;
    float frame_u, frame_v;
};

// include/dynamics/radiative_face.hpp: four separately rounded FP32 operations.
__device__ __forceinline__ float kw78_updated_face(float previous, float phase, float gradient, float dt_rad,
                                                   float inv_spacing, bool negative_outgoing)
{
    if (negative_outgoing ? phase >= 0.0f : phase <= 0.0f) return previous;
    const float dt_phase = __fmul_rn(dt_rad, phase);
    const float tendency = __fmul_rn(dt_phase, gradient);
    const float increment = __fmul_rn(tendency, inv_spacing);
    return __fsub_rn(previous, increment);
}

// V consecutive levels of a field (V = 4: one 16-byte access, where columns and
// field bases allow it; else V = 1).
template <int V>
struct Levels
{
    float v[V];
};

template <int V>
__device__ __forceinline__ Levels<V> load_levels(const float* f)
{
    Levels<V> o;
    if constexpr (V == 4)
    {
        const float4 t = *reinterpret_cast<const float4*>(f);
        o.v[0] = t.x;
        o.v[1] = t.y;
        o.v[2] = t.z;
        o.v[3] = t.w;
    }
    else o.v[0] = *f;
    return o;
}

template <int V>
__device__ __forceinline__ void store_levels(float* f, const Levels<V>& x)
{
    if constexpr (V == 4) *reinterpret_cast<float4*>(f) = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
    else *f = x.v[0];
}

// One lateral axis of the closure: its cells and their stride, the codes of its
// low (west / south) and high (east / north) face, 1 / spacing and the frame's
// velocity along the axis and across it.
struct BoundaryAxis
{
    int n, stride, lo, hi;
    float inv, frame_n, frame_c;
};

// The low (high = false) or high face of one row along an axis, for V levels
// from `base` (the row's cell 0): boundary_conditions_cartesian_cgrid.cpp:927-1121.
// normal and cross are the velocities along and across the axis; hist the
// row's KW78 memory on that face.  The two faces of a row share no cell (n >= 4:
// the low one reads cell 1, or n-2 when periodic, and writes cell 0; the high
// one reads cells 1 and n-3 up and writes n-2 and n-1), except that a periodic
// low face takes the normal velocity of n-2 before the high face writes it:
// bc_axis_face then closes the two in that order in one thread.
template <int V>
__device__ __forceinline__ void bc_low_face(const BoundaryAxis& A, float dt_rad, float* normal, float* cross, float* w,
                                            float* rho, float* p, float* hist, int base)
{
    const bool radiate = A.lo == kBcRadiative && dt_rad > 0.0f;
    const int src = base + (A.lo == kBcPeriodic ? A.n - 2 : 1) * A.stride;
    Levels<V> nl = load_levels<V>(normal + src), cl = load_levels<V>(cross + src), wl = load_levels<V>(w + src);
    const Levels<V> rl = load_levels<V>(rho + src), pl = load_levels<V>(p + src);
    bool store_n = true;
    if (A.lo == kBcRadiative)
    {
        store_n = radiate;
        if (radiate)
        {
            const Levels<V> f = load_levels<V>(hist);
#pragma unroll
            for (int q = 0; q < V; ++q)
            {
                const float up = f.v[q];
                const float phase = __fsub_rn(__fsub_rn(up, A.frame_n), kCStar);
                nl.v[q] = kw78_updated_face(up, phase, __fsub_rn(nl.v[q], up), dt_rad, A.inv, true);
            }
            store_levels<V>(hist, nl);
        }
    }
    else if (A.lo == kBcRigid || A.lo == kBcRigidSlip)
    {
#pragma unroll
        for (int q = 0; q < V; ++q) nl.v[q] = A.frame_n;
    }
    if (A.lo == kBcRigid)
    {
#pragma unroll
        for (int q = 0; q < V; ++q)
        {
            cl.v[q] = A.frame_c;
            wl.v[q] = 0.0f;
        }
    }
    if (store_n) store_levels<V>(normal + base, nl);
    store_levels<V>(cross + base, cl);
    store_levels<V>(w + base, wl);
    store_levels<V>(rho + base, rl);
    store_levels<V>(p + base, pl);
}

template <int V>
__device__ __forceinline__ void bc_high_face(const BoundaryAxis& A, float dt_rad, float* normal, float* cross,
                                             float* w, float* rho, float* p, float* hist, int base)
{
    const bool radiate = A.hi == kBcRadiative && dt_rad > 0.0f;
    const int a = base + (A.n - 2) * A.stride, g = base + (A.n - 1) * A.stride;
    const int src = A.hi == kBcPeriodic ? base + A.stride : a;
    Levels<V> nh = load_levels<V>(normal + src), ch = load_levels<V>(cross + src), wh = load_levels<V>(w + src);
    const Levels<V> rh = load_levels<V>(rho + src), ph = load_levels<V>(p + src);
    if (A.hi != kBcPeriodic)
    {
        bool store_a = true;
        if (A.hi == kBcRigid || A.hi == kBcRigidSlip)
        {
#pragma unroll
            for (int q = 0; q < V; ++q) nh.v[q] = A.frame_n;
        }
        else if (radiate)
        {
            const Levels<V> inner = load_levels<V>(normal + base + (A.n - 3) * A.stride), f = load_levels<V>(hist);
#pragma unroll
            for (int q = 0; q < V; ++q)
            {
                const float up = f.v[q];
                const float phase = __fadd_rn(__fsub_rn(up, A.frame_n), kCStar);
                nh.v[q] = kw78_updated_face(up, phase, __fsub_rn(up, inner.v[q]), dt_rad, A.inv, false);
            }
            store_levels<V>(hist, nh);
        }
        else if (A.hi == kBcZeroGradient) nh = load_levels<V>(normal + base + (A.n - 3) * A.stride);
        else store_a = false;  // radiative without radiation keeps its face
        if (store_a) store_levels<V>(normal + a, nh);
        if (A.hi == kBcRigid)
        {
#pragma unroll
            for (int q = 0; q < V; ++q)
            {
                ch.v[q] = A.frame_c;
                wh.v[q] = 0.0f;
            }
        }
    }
    store_levels<V>(normal + g, nh);
    store_levels<V>(cross + g, ch);
    store_levels<V>(w + g, wh);
    store_levels<V>(rho + g, rh);
    store_levels<V>(p + g, ph);
}

// The low (side = 0) or high (side = 1) face of a row; with a periodic low
// face, side 0 closes both in order and side 1 nothing.
template <int V>
__device__ __forceinline__ void bc_axis_face(const BoundaryAxis& A, int side, float dt_rad, float* normal,
                                             float* cross, float* w, float* rho, float* p, float* hist_lo,
                                             float* hist_hi, int base)
{
    const bool ordered = A.lo == kBcPeriodic;
    if (side == 0) bc_low_face<V>(A, dt_rad, normal, cross, w, rho, p, hist_lo, base);
    if (ordered ? side == 0 : side == 1) bc_high_face<V>(A, dt_rad, normal, cross, w, rho, p, hist_hi, base);
}

// Vertical closure for one (i,j) column: boundary_conditions_cartesian_cgrid.cpp:1124-1175.
__device__ __forceinline__ void bc_vertical_column(const BoundaryParams& B, float* __restrict__ u,
                                                   float* __restrict__ v, float* __restrict__ w, int col)
{
    const Dims d = B.d;
    {
        const int base = col * d.pz;
        if (B.bottom == kBottomNoSlip)
        {
            u[base] = 0.0f;
            v[base] = 0.0f;
        }
        const int kt = base + d.nz - 1, km = base + d.nz - 2;
        w[kt] = (B.top == kTopOpen) ? w[km] : 0.0f;
        u[kt] = u[km];
        v[kt] = v[km];
    }
}

static __global__ void acoustic_bc_vertical_kernel(BoundaryParams B, float* __restrict__ u, float* __restrict__ v,
                                            float* __restrict__ w)
{
    grid_dependency();
    const int cols = B.d.nx * B.d.ny;
    for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < cols; col += gridDim.x * blockDim.x)
        bc_vertical_column(B, u, v, w, col);
}

// Columns whose vertical closure the momentum pass may apply itself: those no
// lateral closure writes or reads.  The others are the perimeter.
__device__ __forceinline__ bool bc_inner_column(const Dims& d, int i, int j)
{
    return i >= 2 && i <= d.nx - 4 && j >= 2 && j <= d.ny - 4;
}

// The closure is independent from level to level except for the top level,
// which takes the one below: a cluster of one to eight CTAs closes a band of
// four levels (the last one up to five) all around the member, with a cluster
// barrier between the reference's steps W,E -> S,N -> vertical instead of a
// launch.  A ring is a few thousand values, so its time is the latency of its
// chain of loads and stores; the cluster spreads a long ring over more SMs.
// One CTA a band -> the cluster: ten closures of 512x512x128 0.47 -> 0.21 ms,
// ten steps of a 256x256x80 member 1.89 -> 1.45 ms.
constexpr int kRingLevels = 4;
constexpr int kRingBlock = 256;

// CTAs a band of `rows` rows takes: one face of a row a thread, up to eight CTAs.
__host__ __device__ __forceinline__ int ring_cluster(int rows)
{
    return 2 * rows <= kRingBlock ? 1 : rows <= kRingBlock ? 2 : rows <= 2 * kRingBlock ? 4 : 8;
}

// The CTA's place in its cluster and the cluster's size (0 and 1 without one).
__device__ __forceinline__ int cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ int cluster_size()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return (int)r;
}
// Barrier of all threads of the cluster; global writes before it are visible
// after it.
__device__ __forceinline__ void cluster_barrier(int size)
{
    if (size == 1) __syncthreads();
    else
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__host__ __device__ __forceinline__ int ring_bands(int nz)
{
    const int bands = (nz + kRingLevels - 1) / kRingLevels;
    return nz % kRingLevels == 1 && bands > 1 ? bands - 1 : bands;  // the top two levels in one band
}

// One band.  vertical: also close the perimeter's columns (their bottom and
// top levels, in the bands that hold them); seed: then fill the KW78 memory
// from the closed faces (seed_radiative_state).  Every thread of the cluster
// calls it.
template <int V>
__device__ __forceinline__ void bc_ring_levels(const BoundaryParams& B, float* u, float* v, float* w, float* rho,
                                               float* p, float* wave, int band, bool vertical, bool seed)
{
    const Dims d = B.d;
    const int size = cluster_size();
    const int first = cluster_rank() * (int)blockDim.x + (int)threadIdx.x, step = size * (int)blockDim.x;
    const int last = ring_bands(d.nz) - 1;
    const int k0 = band * kRingLevels, k1 = band == last ? d.nz : k0 + kRingLevels;
    const int runs = (k1 - k0 + V - 1) / V;
    const int yz = d.ny * d.pz, xz = d.nx * d.pz;
    {
        const BoundaryAxis A{d.nx, d.sx(), B.west, B.east, B.inv_dx, B.frame_u, B.frame_v};
        const int count = d.ny * runs;
        for (int t = first; t < 2 * count; t += step)
        {
            const int side = t >= count, q = t - side * count;
            const int j = q / runs, k = k0 + V * (q - j * runs), r = j * d.pz + k;
            bc_axis_face<V>(A, side, B.dt_rad, u, v, w, rho, p, wave + r, wave + yz + r, d.at(0, j, k));
        }
    }
    cluster_barrier(size);
    {
        const BoundaryAxis A{d.ny, d.sy(), B.south, B.north, B.inv_dy, B.frame_v, B.frame_u};
        float* south = wave + 2 * yz;
        const int count = d.nx * runs;
        for (int t = first; t < 2 * count; t += step)
        {
            const int side = t >= count, q = t - side * count;
            const int i = q / runs, k = k0 + V * (q - i * runs), r = i * d.pz + k;
            bc_axis_face<V>(A, side, B.dt_rad, v, u, w, rho, p, south + r, south + xz + r, d.at(i, 0, k));
        }
    }
    if (vertical && (k0 == 0 || k1 == d.nz))
    {
        cluster_barrier(size);
        // Rows j < loj and j > ny-4 for every i, then i < loi and i > nx-4 between them.
        const int loj = min(2, d.ny - 3), loi = min(2, d.nx - 3);
        const int rows = (loj + 3) * d.nx, sides = loi + 3, mid = d.ny - 3 - loj;
        const int columns = rows + sides * mid;
        const bool bottom = k0 == 0 && B.bottom == kBottomNoSlip, top = k1 == d.nz, open = B.top == kTopOpen;
        // A few columns at a time, their loads together.
        constexpr int kBatch = 4;
        for (int q0 = first; q0 < columns; q0 += kBatch * step)
        {
            int c[kBatch];
            float um[kBatch], vm[kBatch], wm[kBatch];
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
            {
                const int q = min(q0 + b * step, columns - 1);
                int i, j;
                if (q < rows)
                {
                    j = q / d.nx;
                    i = q - j * d.nx;
                    if (j >= loj) j += mid;
                }
                else
                {
                    const int r = q - rows;
                    j = r / sides;
                    i = r - j * sides;
                    j += loj;
                    if (i >= loi) i += d.nx - 3 - loi;
                }
                c[b] = d.at(i, j, 0);
                const int km = c[b] + d.nz - 2;
                um[b] = top ? u[km] : 0.0f;
                vm[b] = top ? v[km] : 0.0f;
                wm[b] = top && open ? w[km] : 0.0f;
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
            {
                if (q0 + b * step >= columns) break;
                if (bottom)
                {
                    u[c[b]] = 0.0f;
                    v[c[b]] = 0.0f;
                    if (d.nz == 2) um[b] = vm[b] = 0.0f;  // the level below the top is the bottom
                }
                if (top)
                {
                    const int kt = c[b] + d.nz - 1;
                    w[kt] = wm[b];
                    u[kt] = um[b];
                    v[kt] = vm[b];
                }
            }
        }
    }
    if (seed)
    {
        cluster_barrier(size);
        const int levels = k1 - k0;
        for (int t = first; t < d.ny * levels; t += step)
        {
            const int j = t / levels, k = k0 + (t - j * levels), r = j * d.pz + k;
            wave[r] = u[d.at(0, j, k)];
            wave[yz + r] = u[d.at(d.nx - 2, j, k)];
        }
        for (int t = first; t < d.nx * levels; t += step)
        {
            const int i = t / levels, k = k0 + (t - i * levels), r = i * d.pz + k;
            wave[2 * yz + r] = v[d.at(i, 0, k)];
            wave[2 * yz + xz + r] = v[d.at(i, d.ny - 2, k)];
        }
    }
}

template <int V>
static __global__ void __launch_bounds__(kRingBlock) acoustic_bc_ring_kernel(BoundaryParams B, float* u, float* v,
                                                                             float* w, float* rho, float* p,
                                                                             float* wave, int vertical)
{
    grid_dependency();
    bc_ring_levels<V>(B, u, v, w, rho, p, wave, (int)blockIdx.x / cluster_size(), vertical != 0, false);
}

// seed_radiative_state (boundary_conditions_cartesian_cgrid.cpp:798-822) for
// history slot r of the west/east (r < ny*nz) and south/north rows.
__device__ __forceinline__ void seed_radiation_row(const Dims& d, const float* __restrict__ u,
                                                   const float* __restrict__ v, float* __restrict__ wave, int r)
{
    const int yz = d.ny * d.nz, xz = d.nx * d.nz;
    {
        if (r < yz)
        {
            const int j = r / d.nz, k = r % d.nz;
            wave[r] = u[d.at(0, j, k)];
            wave[yz + r] = u[d.at(d.nx - 2, j, k)];
        }
        else
        {
            const int q = r - yz;
            const int i = q / d.nz, k = q % d.nz;
            wave[2 * yz + q] = v[d.at(i, 0, k)];
            wave[2 * yz + xz + q] = v[d.at(i, d.ny - 2, k)];
        }
    }
}

static __global__ void acoustic_seed_radiation_kernel(Dims d, const float* __restrict__ u, const float* __restrict__ v,
                                               float* __restrict__ wave)
{
    const int rows = d.ny * d.nz + d.nx * d.nz;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x)
        seed_radiation_row(d, u, v, wave, r);
}

}  // namespace nimbus
