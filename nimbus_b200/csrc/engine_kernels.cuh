// Batched kernels of the member engine: one launch per phase advances that
// phase for every resident member.
//
// Work layout.  Each phase has an item kind (ItemKind: cells, groups of four
// cells, columns, rows along x, bands of levels of the boundary ring).  A
// member's items are cut into tiles of one block and the members' tiles are laid
// end to end; prefix[kind][m] is the first tile of member m.  A persistent
// grid (a few CTAs per SM) strides over the tiles, so the member of a tile is
// uniform across its block and the per-member parameters are warp-broadcast
// loads from the member table.  Members are kept sorted by substep count
// (descending): at substep s the active members are a prefix of the table and
// the launch covers prefix[kind][active_s] tiles -- a ragged ensemble wastes
// no tiles on members that have finished their loop.
//
// Every item runs the same cell function as the per-operation kernels, with
// the member's pointers and parameters, so a member's arithmetic does not
// depend on the batch it shares.
#pragma once

#include "acoustic_kernels.cuh"
#include "acoustic_split.cuh"
#include "bulk_stage.cuh"
#include "physics_kernels.cuh"
#include "relaxation_kernels.cuh"
#include "slow_kernels.cuh"
#include "transport_kernels.cuh"

namespace nimbus
{

enum ItemKind
{
    kItemCells = 0,
    kItemColumns,    // nx*ny columns
    kItemRing,       // bands of levels of the lateral closures (ring_bands), one a CTA
    kItemMarch,      // rows along x: (j, k) positions in blocks times i-chunks (for_member_rows)
    kItemQuads,      // cells in groups of four (the constant-bank acoustic passes and the speed scan)
    kItemKinds
};

constexpr int kQuadTile = kQuadBlock;  // groups of four cells in a kItemQuads tile (one a thread)

constexpr int kEngineScalars = 4;  // theta, qv, qc, qr

struct __align__(16) EngineMember
{
    // Prognostic state and the two ping-pong partners (swapped on the device
    // at the end of the loop / after Kessler, see engine_swap_kernel).
    float *u, *v, *w, *rho, *rho_alt, *p, *theta, *qv, *qc, *qr, *qr_alt;
    // Retained transport context and per-step scratch.
    float *rho_begin, *mfx, *mfy, *mfz, *wave;
    float *sf;        // [3][cells] float4 face fluxes (one lane per scalar)
    float *rl;        // [cells] float4 limiter factors
    float *q4;        // [cells] float4 theta, qv, qc, qr before transport (written by the slow predictor)
    float *k1, *xs;   // [cells] float4 {u, v, w, p}: Heun k1 and predictor state (within sf)
    float *eos;       // EOS candidate pressure
    unsigned* status; // this member's status word (kStatus* bits)
    const double *rho0, *p0, *qv0, *u0, *v0;
    const float2* dp0;
    const float4* eos0;
    FusedParams F;
    BoundaryParams B;
    TransportParams T;  // geometry and flags; the scalar pointers are taken from the fields above
    SlowParams S;
    KesslerParams K;
    double gamma;
    EosSeries eos_series;  // FP32 EOS coefficients binom(gamma, n)
    RelaxTables R;         // end-of-step sponge (all do_* zero: none)
    int close_step;        // end the step with the boundary closure
    int n_substeps;
    int microphysics;
    int march_len;         // i-planes one thread of a marching kernel advances (kItemMarch tiles)
    int march_blocks;      // blocks of blockDim.x (j, k) positions per i-chunk
    int items[kItemKinds];
    long long image_offset;  // first float of this member's block in the engine's state image
};

__device__ __forceinline__ const float* engine_scalar(const EngineMember& M, int s)
{
    return s == 0 ? M.theta : (s == 1 ? M.qv : (s == 2 ? M.qc : M.qr));
}

__device__ __forceinline__ float* engine_scalar_out(const EngineMember& M, int s)
{
    return s == 0 ? M.theta : (s == 1 ? M.qv : (s == 2 ? M.qc : M.qr));
}

// Items per thread in a tile: a tile is kItemsPerThread * blockDim.x
// consecutive items of one member (one item per thread measured fastest:
// more items per thread cost more registers than the shared member lookup
// saves).
constexpr int kItemsPerThread = 1;

// Calls fn(member, item) for every item of the first tiles of a kind.
template <class Fn>
__device__ __forceinline__ void for_member_items(const EngineMember* __restrict__ table,
                                                 const long long* __restrict__ prefix, long long tiles, int kind,
                                                 Fn&& fn)
{
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= prefix[m + 1]) ++m;
        const EngineMember& M = table[m];
        const int count = M.items[kind];
        const int base = (int)((t - prefix[m]) * (kItemsPerThread * blockDim.x)) + (int)threadIdx.x;
#pragma unroll
        for (int q = 0; q < kItemsPerThread; ++q)
        {
            const int item = base + q * (int)blockDim.x;
            if (item < count) fn(M, item);
        }
    }
}

// Calls fn(member, i0, i1, j, k, q) for the rows of the first tiles of
// kItemMarch: a member's (j, k) positions q = j pz + k are cut into blocks of
// blockDim.x (a warp reads 32 consecutive floats of a plane) and its x range
// into chunks of march_len planes; tile = chunk * march_blocks + block.  The
// thread of position q advances the cells (i0 .. i1-1, j, k) of its row.
template <class Fn>
__device__ __forceinline__ void for_member_rows(const EngineMember* __restrict__ table,
                                                const long long* __restrict__ prefix, long long tiles, Fn&& fn)
{
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= prefix[m + 1]) ++m;
        const EngineMember& M = table[m];
        const int local = (int)(t - prefix[m]);
        const int chunk = local / M.march_blocks;
        const int q = (local - chunk * M.march_blocks) * (int)blockDim.x + (int)threadIdx.x;
        const Dims d = M.F.d;
        if (q >= d.sx()) continue;
        int i, j, k;
        decompose(d, q, i, j, k);
        if (k >= d.nz) continue;
        const int i0 = chunk * M.march_len;
        fn(M, i0, min(d.nx, i0 + M.march_len), j, k, q);
    }
}

// ---- Heun slow step -------------------------------------------------------

// Resident CTAs per SM of the slow Heun pair: the reference-precision form at
// 4 of 256 threads (64 registers; four steps of 3.0 million cells at 3 / 4 / 5:
// 1.60 / 1.41 / 1.72 ms), the FP32 form at 5 of kQuadTile threads (96; ten steps of
// 24 members, 17.4 million cells, at 5 / 6 / 7: 9.77 / 9.86 / 9.81 ms).
#ifndef NIMBUS_SLOW_MINB
#define NIMBUS_SLOW_MINB 4
#endif
#ifndef NIMBUS_SLOW_MINB_F32
#define NIMBUS_SLOW_MINB_F32 5
#endif
template <class Policy>
static __global__ void __launch_bounds__(256, 4) engine_slow_predict_kernel(const EngineMember* __restrict__ table,
                                                                  const long long* __restrict__ prefix,
                                                                  long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        slow_predict_packed<Policy>(M.S, M.u, M.v, M.w, M.rho, M.p, M.qv, M.qc, M.qr, M.rho0, M.qv0, M.u0, M.v0,
                                    reinterpret_cast<float4*>(M.k1), reinterpret_cast<float4*>(M.xs), c);
        // The transported scalars do not change before transport: keep their
        // interleaved copy for the transport kernels.
        reinterpret_cast<float4*>(M.q4)[c] = make_float4(M.theta[c], M.qv[c], M.qc[c], M.qr[c]);
    });
}

template <class Policy>
static __global__ void __launch_bounds__(256, 4) engine_slow_correct_kernel(const EngineMember* __restrict__ table,
                                                                  const long long* __restrict__ prefix,
                                                                  long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        slow_correct_packed<Policy>(M.S, reinterpret_cast<const float4*>(M.xs), M.rho, M.qv, M.qc, M.qr, M.rho0,
                                    M.qv0, M.u0, M.v0, reinterpret_cast<const float4*>(M.k1), M.u, M.v, M.w, M.p, c);
    });
}

// The Heun pair with the members' constants in the constant bank (the
// acoustic passes' reason, below: parameters read from the member table sit
// in registers, and the pair spilled at 64 registers).  Each lane's launch
// gets its members' SlowParams and every buffer that does not rotate as one
// __grid_constant__ parameter; density, pressure and rain, which rotate, are
// read from the table.
struct SlowConst
{
    SlowParams S;
    float *u, *v, *w, *theta, *qv, *qc;
    float4 *k1, *xs, *q4;
    const double *rho0, *qv0, *u0, *v0;
};

constexpr int kSlowConstMembers = 64;

struct SlowLaunch
{
    long long prefix[kSlowConstMembers + 1];  // first cell tile of each member
    SlowConst m[kSlowConstMembers];
};
static_assert(sizeof(SlowLaunch) <= 32000, "a kernel parameter block holds at most 32764 bytes");

template <class Policy>
static __global__ void __launch_bounds__(256, NIMBUS_SLOW_MINB) engine_slow_predict_const_kernel(
    const __grid_constant__ SlowLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const SlowConst& A = L.m[m];
        const int c = (int)((t - L.prefix[m]) * blockDim.x) + (int)threadIdx.x;
        if (c >= A.S.d.cells()) continue;
        const EngineMember& M = table[m];
        slow_predict_packed<Policy>(A.S, A.u, A.v, A.w, M.rho, M.p, A.qv, A.qc, M.qr, A.rho0, A.qv0, A.u0, A.v0, A.k1,
                                    A.xs, c);
        A.q4[c] = make_float4(A.theta[c], A.qv[c], A.qc[c], M.qr[c]);
    }
}

template <class Policy>
static __global__ void __launch_bounds__(256, NIMBUS_SLOW_MINB) engine_slow_correct_const_kernel(
    const __grid_constant__ SlowLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const SlowConst& A = L.m[m];
        const int c = (int)((t - L.prefix[m]) * blockDim.x) + (int)threadIdx.x;
        if (c >= A.S.d.cells()) continue;
        const EngineMember& M = table[m];
        slow_correct_packed<Policy>(A.S, A.xs, M.rho, A.qv, A.qc, M.qr, A.rho0, A.qv0, A.u0, A.v0, A.k1, A.u, A.v,
                                    A.w, M.p, c);
    }
}

// The FP32 form, four cells per thread (slow_tendencies_quad): tiles of
// kItemQuads, k1 and the predictor as four planes each.
template <class Policy>
static __global__ void __launch_bounds__(kQuadTile, NIMBUS_SLOW_MINB_F32) engine_slow_predict_quad_kernel(
    const __grid_constant__ SlowLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const SlowConst& A = L.m[m];
        const int n = A.S.d.cells(), c = 4 * ((int)(t - L.prefix[m]) * kQuadTile + (int)threadIdx.x);
        if (c >= n) continue;
        const EngineMember& M = table[m];
        slow_predict_quad(A.S, A.u, A.v, A.w, M.rho, M.p, A.qv, A.qc, M.qr, A.rho0, A.qv0, A.u0, A.v0,
                          reinterpret_cast<float*>(A.k1), reinterpret_cast<float*>(A.xs), (size_t)n, c);
        const Quad th = load_quad(A.theta, c), qv = load_quad(A.qv, c), qc = load_quad(A.qc, c), qr = load_quad(M.qr, c);
#pragma unroll
        for (int q = 0; q < 4; ++q) A.q4[c + q] = make_float4(th.v[q], qv.v[q], qc.v[q], qr.v[q]);
    }
}

template <class Policy>
static __global__ void __launch_bounds__(kQuadTile, NIMBUS_SLOW_MINB_F32) engine_slow_correct_quad_kernel(
    const __grid_constant__ SlowLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const SlowConst& A = L.m[m];
        const int n = A.S.d.cells(), c = 4 * ((int)(t - L.prefix[m]) * kQuadTile + (int)threadIdx.x);
        if (c >= n) continue;
        const EngineMember& M = table[m];
        slow_correct_quad(A.S, reinterpret_cast<const float*>(A.xs), M.rho, A.qv, A.qc, M.qr, A.rho0, A.qv0, A.u0,
                          A.v0, reinterpret_cast<const float*>(A.k1), (size_t)n, A.u, A.v, A.w, M.p, c);
    }
}

// ---- Boundaries and KW78 seed ---------------------------------------------
//
// The density buffer substep s reads (written == false) or writes: substep s
// reads (s even ? rho : rho_alt) and writes the other one.  The boundary
// closure after substep s works on the written buffer; the refresh before the
// loop on the current density.

__device__ __forceinline__ float* engine_density(const EngineMember& M, int s, bool written)
{
    const bool even = (s & 1) == 0;
    return written ? (even ? M.rho_alt : M.rho) : (even ? M.rho : M.rho_alt);
}

// The closure of a band of levels per cluster (bc_ring_levels), one band a
// tile.  refresh 0: inside the acoustic loop, after substep s, with the
// perimeter's vertical closure (the momentum pass closes the inner columns
// itself, fuse_vertical); 1 before the loop, seeding the KW78 memory as well;
// 2 the closing refresh, of the members that ask for it.
static __global__ void __launch_bounds__(kRingBlock) engine_bc_ring_kernel(const EngineMember* __restrict__ table,
                                                                           const long long* __restrict__ prefix, int s,
                                                                           int refresh)
{
    grid_dependency();
    const int t = (int)blockIdx.x / cluster_size();
    int m = 0;
    while (t >= prefix[m + 1]) ++m;
    const EngineMember& M = table[m];
    if (refresh == 2 && !M.close_step) return;
    BoundaryParams B = M.B;
    if (refresh) B.dt_rad = 0.0f;
    bc_ring_levels<4>(B, M.u, M.v, M.w, refresh ? M.rho : engine_density(M, s, true), M.p, M.wave,
                      t - (int)prefix[m], true, refresh == 1);
}

// refresh: 1 before the acoustic loop, 2 the closing refresh at the end of the
// step (members with close_step only).
static __global__ void __launch_bounds__(256) engine_bc_vertical_kernel(const EngineMember* __restrict__ table,
                                                                 const long long* __restrict__ prefix,
                                                                 long long tiles, int refresh)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemColumns, [&](const EngineMember& M, int col) {
        if (refresh == 2 && !M.close_step) return;
        bc_vertical_column(M.B, M.u, M.v, M.w, col);
    });
}

// ---- Acoustic substep (split form, u/v/w in place, rho ping-pong) ---------

template <class Policy>
static __global__ void __launch_bounds__(256, 5) engine_continuity_kernel(const EngineMember* __restrict__ table,
                                                                const long long* __restrict__ prefix,
                                                                long long tiles, int s)
{
    grid_dependency();
    const bool first = s == 0;
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        unsigned flags = 0;
        continuity_eos_cell<Policy>(M.F, engine_density(M, s, false), M.u, M.v, M.w, M.theta, M.rho0, M.eos0,
                                    engine_density(M, s, true), M.p, nullptr, M.mfx, M.mfy, M.mfz, c, flags, first,
                                    first ? M.rho_begin : nullptr);
        if (flags) atomicOr(M.status, flags);
    });
}

template <class Policy>
static __global__ void __launch_bounds__(256) engine_momentum_kernel(const EngineMember* __restrict__ table,
                                                              const long long* __restrict__ prefix, long long tiles,
                                                              int s)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        const int vertical = kFuseVertical | (M.B.bottom == kBottomNoSlip ? kFuseNoSlipBottom : 0) |
                             (M.B.top == kTopOpen ? kFuseOpenTop : 0);
        momentum_cell<Policy>(M.F, engine_density(M, s, true), M.p, M.p0, M.dp0, M.u, M.v, M.w, M.u, M.v, M.w, c,
                              vertical);
    });
}

// The same two passes marching along x (continuity_eos_march, momentum_march):
// one thread per (j, k) row segment of march_len cells.
#ifndef NIMBUS_MARCH_MINB
#define NIMBUS_MARCH_MINB 4
#endif
template <class Policy>
static __global__ void __launch_bounds__(256, NIMBUS_MARCH_MINB) engine_continuity_march_kernel(const EngineMember* __restrict__ table,
                                                                      const long long* __restrict__ prefix,
                                                                      long long tiles, int s)
{
    grid_dependency();
    const bool first = s == 0;
    for_member_rows(table, prefix, tiles, [&](const EngineMember& M, int i0, int i1, int j, int k, int q) {
        unsigned flags = 0;
        continuity_eos_march<Policy>(M.F, engine_density(M, s, false), M.u, M.v, M.w, M.theta, M.rho0, M.eos0,
                                     engine_density(M, s, true), M.p, M.mfx, M.mfy, M.mfz, i0, i1, j, k, q, flags,
                                     first, first ? M.rho_begin : nullptr);
        if (flags) atomicOr(M.status, flags);
    });
}

template <class Policy>
static __global__ void __launch_bounds__(256) engine_momentum_march_kernel(const EngineMember* __restrict__ table,
                                                                    const long long* __restrict__ prefix,
                                                                    long long tiles, int s)
{
    grid_dependency();
    for_member_rows(table, prefix, tiles, [&](const EngineMember& M, int i0, int i1, int j, int k, int q) {
        const int vertical = kFuseVertical | (M.B.bottom == kBottomNoSlip ? kFuseNoSlipBottom : 0) |
                             (M.B.top == kTopOpen ? kFuseOpenTop : 0);
        momentum_march<Policy>(M.F, engine_density(M, s, true), M.p, M.p0, M.dp0, M.u, M.v, M.w, i0, i1, j, k, q,
                               vertical);
    });
}

// ---- Acoustic passes with the members' constants in the constant bank ----
//
// A kernel that reads a member's parameters and pointers from the member
// table holds them in registers (about 50 values for continuity), which caps
// it at 5-6 resident CTAs per SM; the per-operation kernels take the same
// values from the constant bank as instruction operands and run at full
// occupancy with 32 registers.  So each launch of a lane gets its members'
// constants as one kernel parameter (__grid_constant__, the constant bank):
// the parameter blocks and every buffer that does not rotate.  The rotating
// buffers (density ping-pong, pressure) are read from the member table.
struct AcousticConst
{
    FusedParams F;
    float *u, *v, *w, *theta, *mfx, *mfy, *mfz, *rho_begin;
    unsigned* status;
    const double *rho0, *p0;
    const float2* dp0;
    const float4* eos0;
    int vertical;  // kFuse* bits of the momentum pass
    int march_len, march_blocks;  // the marching forms' row tiling (kItemMarch)
};

constexpr int kConstMembers = 64;  // members one launch can carry in its parameter

// The part of the parameter block every member of a launch holds alike (field
// bounds, EOS exponent and coefficients, frame velocity, top condition).  A
// member's own block is indexed by the member, so each value it supplies is an
// indexed constant load per cell; from here the kernel takes them as operands
// at fixed constant-bank offsets.
struct AcousticShared
{
    double gamma, frame_u, frame_v;
    float rho_min, rho_max, p_min, p_max, p_ref_fallback, frame_u_f, frame_v_f;
    int top_open;
    float eos_c[6];
};

inline AcousticShared acoustic_shared_of(const FusedParams& F)
{
    AcousticShared S{};
    S.gamma = F.gamma;
    S.frame_u = F.frame_u;
    S.frame_v = F.frame_v;
    S.rho_min = F.rho_min;
    S.rho_max = F.rho_max;
    S.p_min = F.p_min;
    S.p_max = F.p_max;
    S.p_ref_fallback = F.p_ref_fallback;
    S.frame_u_f = F.frame_u_f;
    S.frame_v_f = F.frame_v_f;
    S.top_open = F.top_open;
    for (int n = 0; n < 6; ++n) S.eos_c[n] = F.eos_c[n];
    return S;
}

// A member's block with the shared values read from S (bitwise equal to its
// own: the launch checks that before choosing a kernel that uses this).
__device__ __forceinline__ FusedParams with_shared(const FusedParams& F, const AcousticShared& S)
{
    FusedParams P = F;
    P.gamma = S.gamma;
    P.frame_u = S.frame_u;
    P.frame_v = S.frame_v;
    P.rho_min = S.rho_min;
    P.rho_max = S.rho_max;
    P.p_min = S.p_min;
    P.p_max = S.p_max;
    P.p_ref_fallback = S.p_ref_fallback;
    P.frame_u_f = S.frame_u_f;
    P.frame_v_f = S.frame_v_f;
    P.top_open = S.top_open;
    for (int n = 0; n < 6; ++n) P.eos_c[n] = S.eos_c[n];
    return P;
}

struct AcousticLaunch
{
    long long prefix[kConstMembers + 1];        // first cell tile of each member
    int quad_prefix[kConstMembers + 1];         // first quad tile of each member (a lane's tiles fit 32 bits)
    long long march_prefix[kConstMembers + 1];  // first row tile of each member (marching forms)
    AcousticConst m[kConstMembers];
    int bulk_sy4;                               // the members' largest nz rounded up to 4 (bulk-staged forms)
    AcousticShared shared;                      // every member's shared values (kernels with kShared)
};
static_assert(sizeof(AcousticLaunch) <= 32000, "a kernel parameter block holds at most 32764 bytes");

// Calls fn(A, M, c) for the first tiles' cells: kCells = 4, one group of four
// cells per thread of a kItemQuads tile; kCells = 1, one cell per thread, a CTA
// taking a quarter of a tile (small lanes, kQuadCells).
template <int kCells, class Fn>
__device__ __forceinline__ void for_const_cells(const AcousticLaunch& L, const EngineMember* __restrict__ table,
                                                int tiles, Fn&& fn)
{
    constexpr int kParts = 4 / kCells;
    int m = 0;
    for (int t = blockIdx.x; t < kParts * tiles; t += gridDim.x)
    {
        while (t >= kParts * L.quad_prefix[m + 1]) ++m;
        const AcousticConst& A = L.m[m];
        const int c = kCells * ((t - kParts * L.quad_prefix[m]) * kQuadTile + (int)threadIdx.x);
        if (c >= A.F.d.cells()) continue;
        fn(A, table[m], c);
    }
}

// kFirst: the first substep of the step (the retained fluxes are written, not
// accumulated, and the beginning density is kept).
// kShared: every member's shared values equal L.shared (acoustic_shared_of).
template <class Policy, bool kFirst, bool kShared, int kCells>
static __global__ void __launch_bounds__(kQuadTile, kQuadCtas<Policy>) engine_continuity_const_kernel(const __grid_constant__ AcousticLaunch L,
                                                                      const EngineMember* __restrict__ table,
                                                                      long long tiles, int s)
{
    grid_dependency();
    const bool even = (s & 1) == 0;
    for_const_cells<kCells>(L, table, (int)tiles, [&](const AcousticConst& A, const EngineMember& M, int c) {
        unsigned flags = 0;
        const FusedParams F = kShared ? with_shared(A.F, L.shared) : A.F;
        float* const before = even ? M.rho : M.rho_alt;
        float* const after = even ? M.rho_alt : M.rho;
        float* const begin = kFirst ? A.rho_begin : nullptr;
        if constexpr (kCells == 4)
            continuity_eos_quad<Policy>(F, before, A.u, A.v, A.w, A.theta, A.rho0, A.eos0, after, M.p, A.mfx, A.mfy,
                                        A.mfz, c, flags, kFirst, begin);
        else
            continuity_eos_cell<Policy>(F, before, A.u, A.v, A.w, A.theta, A.rho0, A.eos0, after, M.p, nullptr, A.mfx,
                                        A.mfy, A.mfz, c, flags, kFirst, begin);
        if (flags) atomicOr(A.status, flags);
    });
}

template <class Policy, int kCells>
static __global__ void __launch_bounds__(kQuadTile, kQuadCtas<Policy>) engine_momentum_const_kernel(const __grid_constant__ AcousticLaunch L,
                                                                    const EngineMember* __restrict__ table,
                                                                    long long tiles, int s)
{
    grid_dependency();
    const bool even = (s & 1) == 0;
    for_const_cells<kCells>(L, table, (int)tiles, [&](const AcousticConst& A, const EngineMember& M, int c) {
        const float* rho = even ? M.rho_alt : M.rho;
        if constexpr (kCells == 4)
            momentum_quad<Policy>(A.F, rho, M.p, A.p0, A.dp0, A.u, A.v, A.w, A.u, A.v, A.w, c, A.vertical);
        else
            momentum_cell<Policy>(A.F, rho, M.p, A.p0, A.dp0, A.u, A.v, A.w, A.u, A.v, A.w, c, A.vertical);
    });
}

// The marching passes with the members' constants in the constant bank.
#ifndef NIMBUS_CMARCH_MINB
#define NIMBUS_CMARCH_MINB 5
#endif
template <class Fn>
__device__ __forceinline__ void for_const_rows(const AcousticLaunch& L, const EngineMember* __restrict__ table,
                                               long long tiles, Fn&& fn)
{
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.march_prefix[m + 1]) ++m;
        const AcousticConst& A = L.m[m];
        const int local = (int)(t - L.march_prefix[m]);
        const int chunk = local / A.march_blocks;
        const int q = (local - chunk * A.march_blocks) * (int)blockDim.x + (int)threadIdx.x;
        const Dims d = A.F.d;
        if (q >= d.sx()) continue;
        int i, j, k;
        decompose(d, q, i, j, k);
        if (k >= d.nz) continue;
        const int i0 = chunk * A.march_len;
        fn(A, table[m], i0, min(d.nx, i0 + A.march_len), j, k, q);
    }
}

template <class Policy, bool kFirst>
static __global__ void __launch_bounds__(256, NIMBUS_CMARCH_MINB) engine_continuity_cmarch_kernel(
    const __grid_constant__ AcousticLaunch L, const EngineMember* __restrict__ table, long long tiles, int s)
{
    grid_dependency();
    const bool even = (s & 1) == 0;
    for_const_rows(L, table, tiles, [&](const AcousticConst& A, const EngineMember& M, int i0, int i1, int j, int k,
                                        int q) {
        unsigned flags = 0;
        continuity_eos_march<Policy>(A.F, even ? M.rho : M.rho_alt, A.u, A.v, A.w, A.theta, A.rho0, A.eos0,
                                     even ? M.rho_alt : M.rho, M.p, A.mfx, A.mfy, A.mfz, i0, i1, j, k, q, flags, kFirst,
                                     kFirst ? A.rho_begin : nullptr);
        if (flags) atomicOr(A.status, flags);
    });
}

template <class Policy>
static __global__ void __launch_bounds__(256, NIMBUS_CMARCH_MINB) engine_momentum_cmarch_kernel(
    const __grid_constant__ AcousticLaunch L, const EngineMember* __restrict__ table, long long tiles, int s)
{
    grid_dependency();
    const bool even = (s & 1) == 0;
    for_const_rows(L, table, tiles, [&](const AcousticConst& A, const EngineMember& M, int i0, int i1, int j, int k,
                                        int q) {
        momentum_march<Policy>(A.F, even ? M.rho_alt : M.rho, M.p, A.p0, A.dp0, A.u, A.v, A.w, i0, i1, j, k, q,
                               A.vertical);
    });
}

// The same two passes with each tile's stencil data staged in shared memory
// by bulk copies (bulk_stage.cuh).  A tile is 256 consecutive cells of one
// member (one per thread); its stencils read, per field, the tile itself and
// the tile shifted by the neighbour strides, each a contiguous run of cells,
// so one CTA stages a tile with a handful of bulk copies issued by one thread
// and keeps kBulkStages tiles in flight while it computes.  Each cell's
// arithmetic is the one-cell form's, on the same values.
constexpr int kBulkStages = 4;
constexpr int kBulkTile = 256;
constexpr int kBulkCap = kBulkTile + 8;  // a run of the tile's length widened to 16-byte units
constexpr int kBulkBarrierBytes = 64;
#ifndef NIMBUS_BULK_MINB
#define NIMBUS_BULK_MINB 4
#endif

// Floats of one continuity stage: eleven runs, R0 (rho at -x), R1 (rho at
// the tile, +-1, +-y), R2 (rho at +x), U1 (u at the tile), U0 (u at -x), V (v
// at the tile and -y), W (w at the tile and -1), TH, MX, MY, MZ.
__host__ __device__ constexpr int continuity_stage_floats(int sy4) { return 11 * kBulkCap + 3 * sy4; }
// Floats of one momentum stage: RA, PA (tile, +1, +y), RB, PB (+x), U, V, W.
__host__ __device__ constexpr int momentum_stage_floats(int sy4) { return 7 * kBulkCap + 2 * sy4; }

// Slot offsets of the two stage layouts (floats), the last entry the stage end.
__host__ __device__ constexpr int continuity_slot(int slot, int sy4)
{
    // R0, R1 (+2 sy4), R2, U1, U0, V (+sy4), W, TH, MX, MY, MZ
    return slot * kBulkCap + (slot >= 2 ? 2 * sy4 : 0) + (slot >= 6 ? sy4 : 0);
}
__host__ __device__ constexpr int momentum_slot(int slot, int sy4)
{
    // RA (+sy4), PA (+sy4), RB, PB, U, V, W
    return slot * kBulkCap + (slot >= 1 ? sy4 : 0) + (slot >= 2 ? sy4 : 0);
}
static_assert(continuity_slot(11, 8) == continuity_stage_floats(8) && continuity_slot(11, 64) == continuity_stage_floats(64),
              "continuity stage layout");
static_assert(momentum_slot(7, 8) == momentum_stage_floats(8) && momentum_slot(7, 64) == momentum_stage_floats(64),
              "momentum stage layout");

__device__ __forceinline__ unsigned run_bytes(const CellRun& r) { return r.hi > r.lo ? 4u * (r.hi - r.lo) : 0u; }

__device__ __forceinline__ void stage_run(float* dst, const float* field, const CellRun& r, uint64_t* bar)
{
    if (r.hi > r.lo) bulk_copy_g2s(dst, field + r.lo, run_bytes(r), bar);
}

struct ContinuityRuns
{
    CellRun r0, r1, r2, t, v, w;  // r0 also serves u at -x; t the tile (u, theta, mx, my, mz)
};

__device__ __forceinline__ ContinuityRuns continuity_runs(int c0, int c1, int n, int sx, int sy)
{
    ContinuityRuns R;
    R.r0 = cell_run((long long)c0 - sx, (long long)c1 - sx, n);
    R.r1 = cell_run((long long)c0 - sy, (long long)c1 + sy, n);
    R.r2 = cell_run((long long)c0 + sx, (long long)c1 + sx, n);
    R.t = cell_run(c0, c1, n);
    R.v = cell_run((long long)c0 - sy, c1, n);
    R.w = cell_run((long long)c0 - 1, c1, n);
    return R;
}

struct MomentumRuns
{
    CellRun a, b, t;  // a: tile .. +y (rho, p); b: +x (rho, p); t: the tile (u, v, w)
};

__device__ __forceinline__ MomentumRuns momentum_runs(int c0, int c1, int n, int sx, int sy)
{
    MomentumRuns R;
    R.a = cell_run(c0, (long long)c1 + sy, n);
    R.b = cell_run((long long)c0 + sx, (long long)c1 + sx, n);
    R.t = cell_run(c0, c1, n);
    return R;
}

// Ends a CTA whose stage wait timed out: the member's status gets
// kStatusStagingTimeout and thread 0 waits (bounded) for the copies of the
// stages it issued that are still outstanding before the CTA leaves.
__device__ __forceinline__ void bulk_abandon(uint64_t* bar, unsigned parity_bits, int pending, unsigned* status)
{
    if (threadIdx.x == 0)
    {
        atomicOr(status, kStatusStagingTimeout);
        for (int q = 0; q < kBulkStages; ++q)
            if (pending & (1 << q)) (void)mbar_wait(&bar[q], (parity_bits >> q) & 1u);
    }
    __syncthreads();
}

template <class Policy, bool kFirst>
static __global__ void __launch_bounds__(256, NIMBUS_BULK_MINB) engine_continuity_bulk_kernel(const __grid_constant__ AcousticLaunch L,
                                                                     const EngineMember* __restrict__ table,
                                                                     long long tiles, int s)
{
    grid_dependency();
    extern __shared__ __align__(16) unsigned char bulk_smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(bulk_smem);
    float* stages = reinterpret_cast<float*>(bulk_smem + kBulkBarrierBytes);
    const int sy4 = L.bulk_sy4;
    const int o_r1 = continuity_slot(1, sy4), o_r2 = continuity_slot(2, sy4), o_u1 = continuity_slot(3, sy4),
              o_u0 = continuity_slot(4, sy4), o_v = continuity_slot(5, sy4), o_w = continuity_slot(6, sy4),
              o_th = continuity_slot(7, sy4), o_mx = continuity_slot(8, sy4), o_my = continuity_slot(9, sy4),
              o_mz = continuity_slot(10, sy4);
    const int stage_floats = continuity_stage_floats(sy4);
    const bool even = (s & 1) == 0;
    if (threadIdx.x == 0)
    {
        for (int q = 0; q < kBulkStages; ++q) mbar_init(&bar[q], 1);
        mbar_init_fence();
    }
    __syncthreads();

    int pm = 0;                        // the producer's member cursor
    unsigned parity = 0;               // bit q: the parity of stage q's next phase
    int pending = 0;                   // stages issued and not yet consumed (thread 0's view)
    // Thread 0: stage tile t into stage q.
    auto issue = [&](long long t, int q) {
        while (t >= L.prefix[pm + 1]) ++pm;
        const AcousticConst& A = L.m[pm];
        const Dims d = A.F.d;
        const int n = d.cells();
        const int c0 = (int)((t - L.prefix[pm]) * kBulkTile), c1 = min(c0 + kBulkTile, n);
        const EngineMember& M = table[pm];
        const float* rho = even ? M.rho : M.rho_alt;
        const ContinuityRuns R = continuity_runs(c0, c1, n, d.sx(), d.sy());
        unsigned bytes = 2 * run_bytes(R.r0) + run_bytes(R.r1) + run_bytes(R.r2) + 2 * run_bytes(R.t) +
                         run_bytes(R.v) + run_bytes(R.w);
        if (!kFirst) bytes += 3 * run_bytes(R.t);
        float* S = stages + q * stage_floats;
        mbar_arrive_expect_tx(&bar[q], bytes);
        stage_run(S, rho, R.r0, &bar[q]);
        stage_run(S + o_r1, rho, R.r1, &bar[q]);
        stage_run(S + o_r2, rho, R.r2, &bar[q]);
        stage_run(S + o_u1, A.u, R.t, &bar[q]);
        stage_run(S + o_u0, A.u, R.r0, &bar[q]);
        stage_run(S + o_v, A.v, R.v, &bar[q]);
        stage_run(S + o_w, A.w, R.w, &bar[q]);
        stage_run(S + o_th, A.theta, R.t, &bar[q]);
        if (!kFirst)
        {
            stage_run(S + o_mx, A.mfx, R.t, &bar[q]);
            stage_run(S + o_my, A.mfy, R.t, &bar[q]);
            stage_run(S + o_mz, A.mfz, R.t, &bar[q]);
        }
        pending |= 1 << q;
    };
    const long long stride = gridDim.x;
    if (threadIdx.x == 0)
        for (int q = 0; q < kBulkStages; ++q)
        {
            const long long t = blockIdx.x + q * stride;
            if (t < tiles) issue(t, q);
        }

    int m = 0;
    int it = 0;
    for (long long t = blockIdx.x; t < tiles; t += stride, ++it)
    {
        const int q = it % kBulkStages;
        while (t >= L.prefix[m + 1]) ++m;
        const AcousticConst& A = L.m[m];
        const bool ok = mbar_wait(&bar[q], (parity >> q) & 1u);
        if (ok)
        {
            const Dims d = A.F.d;
            const int n = d.cells(), sx = d.sx(), sy = d.sy();
            const int c0 = (int)((t - L.prefix[m]) * kBulkTile), c1 = min(c0 + kBulkTile, n);
            const int c = c0 + (int)threadIdx.x;
            if (c < c1)
            {
                const ContinuityRuns R = continuity_runs(c0, c1, n, sx, sy);
                const float* S = stages + q * stage_floats;
                int i, j, k;
                decompose(d, c, i, j, k);
                if (k < d.nz)
                {
                const bool xlo = i >= 1, xhi = i < d.nx - 1, ylo = j >= 1, yhi = j < d.ny - 1;
                const bool zlo = k > 0, zhi = k + 1 < d.nz;
                const float* r1 = S + o_r1 + (c - R.r1.lo);  // rho at the cell
                ContinuityStencil st;
                st.rho_c = r1[0];
                st.rxp = xhi ? S[o_r2 + (c + sx - R.r2.lo)] : st.rho_c;
                st.rxm = xlo ? S[c - sx - R.r0.lo] : st.rho_c;
                st.ryp = yhi ? r1[sy] : st.rho_c;
                st.rym = ylo ? r1[-sy] : st.rho_c;
                st.rzp = zhi ? r1[1] : st.rho_c;
                st.rzm = zlo ? r1[-1] : st.rho_c;
                const int ct = c - R.t.lo;
                st.uc = S[o_u1 + ct];
                st.uxm = xlo ? S[o_u0 + c - sx - R.r0.lo] : st.uc;
                st.vc = S[o_v + c - R.v.lo];
                st.vym = ylo ? S[o_v + c - sy - R.v.lo] : st.vc;
                st.wc = S[o_w + c - R.w.lo];
                st.wzm = zlo ? S[o_w + c - 1 - R.w.lo] : st.wc;
                st.th = S[o_th + ct];
                st.mx = kFirst ? 0.0f : S[o_mx + ct];
                st.my = kFirst ? 0.0f : S[o_my + ct];
                st.mz = kFirst ? 0.0f : S[o_mz + ct];
                const EngineMember& M = table[m];
                unsigned flags = 0;
                continuity_eos_values<Policy>(A.F, st, i, j, k, c, A.rho0, A.eos0, even ? M.rho_alt : M.rho, M.p,
                                              nullptr, A.mfx, A.mfy, A.mfz, flags, kFirst,
                                              kFirst ? A.rho_begin : nullptr);
                if (flags) atomicOr(A.status, flags);
                }
            }
        }
        // Every thread is done with stage q (and agrees whether its wait
        // completed) before it is refilled.
        if (!__syncthreads_and(ok))
        {
            bulk_abandon(bar, parity, pending, A.status);
            return;
        }
        parity ^= 1u << q;
        if (threadIdx.x == 0)
        {
            pending &= ~(1 << q);
            const long long next = t + kBulkStages * stride;
            if (next < tiles) issue(next, q);
        }
    }
}

template <class Policy>
static __global__ void __launch_bounds__(256, NIMBUS_BULK_MINB) engine_momentum_bulk_kernel(const __grid_constant__ AcousticLaunch L,
                                                                   const EngineMember* __restrict__ table,
                                                                   long long tiles, int s)
{
    grid_dependency();
    extern __shared__ __align__(16) unsigned char bulk_smem[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(bulk_smem);
    float* stages = reinterpret_cast<float*>(bulk_smem + kBulkBarrierBytes);
    const int sy4 = L.bulk_sy4;
    const int o_pa = momentum_slot(1, sy4), o_rb = momentum_slot(2, sy4), o_pb = momentum_slot(3, sy4),
              o_u = momentum_slot(4, sy4), o_v = momentum_slot(5, sy4), o_w = momentum_slot(6, sy4);
    const int stage_floats = momentum_stage_floats(sy4);
    const bool even = (s & 1) == 0;
    if (threadIdx.x == 0)
    {
        for (int q = 0; q < kBulkStages; ++q) mbar_init(&bar[q], 1);
        mbar_init_fence();
    }
    __syncthreads();

    int pm = 0;
    unsigned parity = 0;
    int pending = 0;
    auto issue = [&](long long t, int q) {
        while (t >= L.prefix[pm + 1]) ++pm;
        const AcousticConst& A = L.m[pm];
        const Dims d = A.F.d;
        const int n = d.cells();
        const int c0 = (int)((t - L.prefix[pm]) * kBulkTile), c1 = min(c0 + kBulkTile, n);
        const EngineMember& M = table[pm];
        const float* rho = even ? M.rho_alt : M.rho;
        const MomentumRuns R = momentum_runs(c0, c1, n, d.sx(), d.sy());
        const unsigned bytes = 2 * run_bytes(R.a) + 2 * run_bytes(R.b) + 3 * run_bytes(R.t);
        float* S = stages + q * stage_floats;
        mbar_arrive_expect_tx(&bar[q], bytes);
        stage_run(S, rho, R.a, &bar[q]);
        stage_run(S + o_pa, M.p, R.a, &bar[q]);
        stage_run(S + o_rb, rho, R.b, &bar[q]);
        stage_run(S + o_pb, M.p, R.b, &bar[q]);
        stage_run(S + o_u, A.u, R.t, &bar[q]);
        stage_run(S + o_v, A.v, R.t, &bar[q]);
        stage_run(S + o_w, A.w, R.t, &bar[q]);
        pending |= 1 << q;
    };
    const long long stride = gridDim.x;
    if (threadIdx.x == 0)
        for (int q = 0; q < kBulkStages; ++q)
        {
            const long long t = blockIdx.x + q * stride;
            if (t < tiles) issue(t, q);
        }

    int m = 0;
    int it = 0;
    for (long long t = blockIdx.x; t < tiles; t += stride, ++it)
    {
        const int q = it % kBulkStages;
        while (t >= L.prefix[m + 1]) ++m;
        const AcousticConst& A = L.m[m];
        const bool ok = mbar_wait(&bar[q], (parity >> q) & 1u);
        if (ok)
        {
            const Dims d = A.F.d;
            const int n = d.cells(), sx = d.sx(), sy = d.sy();
            const int c0 = (int)((t - L.prefix[m]) * kBulkTile), c1 = min(c0 + kBulkTile, n);
            const int c = c0 + (int)threadIdx.x;
            if (c < c1)
            {
                const MomentumRuns R = momentum_runs(c0, c1, n, sx, sy);
                const float* S = stages + q * stage_floats;
                int i, j, k;
                decompose(d, c, i, j, k);
                const bool interior = i >= 1 && i < d.nx - 1 && j >= 1 && j < d.ny - 1 && k < d.nz - 1;
                const float* ra = S + (c - R.a.lo);  // rho at the cell
                const float* pa = S + o_pa + (c - R.a.lo);
                MomentumStencil st;
                st.rc = ra[0];
                st.pc = pa[0];
                st.rx = interior ? S[o_rb + (c + sx - R.b.lo)] : st.rc;
                st.px = interior ? S[o_pb + (c + sx - R.b.lo)] : st.pc;
                st.ry = interior ? ra[sy] : st.rc;
                st.py = interior ? pa[sy] : st.pc;
                st.rz = interior ? ra[1] : st.rc;
                st.pz = interior ? pa[1] : st.pc;
                const int ct = c - R.t.lo;
                st.uc = S[o_u + ct];
                st.vc = S[o_v + ct];
                st.wc = S[o_w + ct];
                if (k < d.nz) momentum_values<Policy>(A.F, st, i, j, k, c, A.p0, A.dp0, A.u, A.v, A.w, A.vertical);
            }
        }
        if (!__syncthreads_and(ok))
        {
            bulk_abandon(bar, parity, pending, A.status);
            return;
        }
        parity ^= 1u << q;
        if (threadIdx.x == 0)
        {
            pending &= ~(1 << q);
            const long long next = t + kBulkStages * stride;
            if (next < tiles) issue(next, q);
        }
    }
}

// ---- state image ----------------------------------------------------------
// A member's nine prognostic fields back to back (u, v, w, rho, p, theta, qv,
// qc, qr, each nx ny nz floats without padding), the host's form of a state.
// gather = 0 scatters an image into the member's current buffers, gather = 1
// collects them into it; only the fields whose bits are set.
__device__ __forceinline__ void image_cell(const EngineMember& M, float* __restrict__ image, int c, int gather,
                                           unsigned fields)
{
    int i, j, k;
    const Dims d = M.F.d;
    decompose(d, c, i, j, k);
    if (k >= d.nz) return;
    const long long n = (long long)d.nx * d.ny * d.nz;
    float* blk = image + (long long)(i * d.ny + j) * d.nz + k;
    float* const field[9] = {M.u, M.v, M.w, M.rho, M.p, M.theta, M.qv, M.qc, M.qr};
    float x[9];
    if (gather)
    {
#pragma unroll
        for (int f = 0; f < 9; ++f)
            if (fields >> f & 1u) x[f] = field[f][c];
#pragma unroll
        for (int f = 0; f < 9; ++f)
            if (fields >> f & 1u) blk[f * n] = x[f];
    }
    else
    {
#pragma unroll
        for (int f = 0; f < 9; ++f)
            if (fields >> f & 1u) x[f] = blk[f * n];
#pragma unroll
        for (int f = 0; f < 9; ++f)
            if (fields >> f & 1u) field[f][c] = x[f];
    }
}

// The engine's state image: every member's from image + image_offset; one
// coalesced pass over all cells of all members.
static __global__ void __launch_bounds__(256) engine_image_kernel(const EngineMember* __restrict__ table,
                                                                  const long long* __restrict__ prefix,
                                                                  long long tiles, float* __restrict__ image,
                                                                  int gather)
{
    for_member_items(table, prefix, tiles, kItemCells,
                     [&](const EngineMember& M, int c) { image_cell(M, image + M.image_offset, c, gather, ~0u); });
}

// One member's image (its table entry by value, before or beside the table).
static __global__ void __launch_bounds__(256) member_image_kernel(const __grid_constant__ EngineMember M,
                                                                  float* __restrict__ image, int gather,
                                                                  unsigned fields)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < M.items[kItemCells]; c += gridDim.x * blockDim.x)
        image_cell(M, image, c, gather, fields);
}

// Pointer rotation after the acoustic loop (rho: with an odd substep count
// the final density sits in the partner) and at the end of the step (qr after
// Kessler; p and the EOS candidate, which publishes the projection).
static __global__ void engine_swap_kernel(EngineMember* table, int members, int which)
{
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= members) return;
    EngineMember& M = table[m];
    if (which == 0)
    {
        if (M.n_substeps & 1)
        {
            float* t = M.rho;
            M.rho = M.rho_alt;
            M.rho_alt = t;
        }
    }
    else
    {
        if (M.microphysics)
        {
            float* t = M.qr;
            M.qr = M.qr_alt;
            M.qr_alt = t;
        }
        if (!(*M.status & kStatusInvalidEos))
        {
            float* t = M.p;
            M.p = M.eos;
            M.eos = t;
        }
    }
}

// ---- Transport (every scalar of a cell in one thread) -----------------------

template <bool kFp32>
// Resident CTAs per SM of the face-flux pass: the FP32 form at 5 (48
// registers; ten steps of 24 members, 17.4 million cells, at 4 / 5 / 6: 5.68 /
// 5.38 / 5.59 ms), the reference-precision form at 4 (64; four
// steps of 3.0 million cells at 2 / 3 / 4 / 5: 1.14 / 0.94 / 0.88 / 0.93 ms).
#ifndef NIMBUS_FACES_MINB
#define NIMBUS_FACES_MINB 4
#endif
#ifndef NIMBUS_FACES_MINB_F32
#define NIMBUS_FACES_MINB_F32 5
#endif
static __global__ void __launch_bounds__(256, NIMBUS_FACES_MINB) engine_transport_faces_kernel(const EngineMember* __restrict__ table,
                                                                            const long long* __restrict__ prefix,
                                                                            long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        transport_faces_cell4<kFp32>(M.T, reinterpret_cast<const float4*>(M.q4), M.mfx, M.mfy, M.mfz,
                                     reinterpret_cast<float4*>(M.sf), c);
    });
}

template <bool kFp32>
static __global__ void __launch_bounds__(256) engine_transport_limiter_kernel(const EngineMember* __restrict__ table,
                                                                              const long long* __restrict__ prefix,
                                                                              long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        transport_limiter_cell4<kFp32>(M.T, reinterpret_cast<const float4*>(M.q4), M.rho_begin,
                                       reinterpret_cast<const float4*>(M.sf), reinterpret_cast<float4*>(M.rl), c);
    });
}

template <bool kFp32>
static __global__ void __launch_bounds__(256) engine_transport_update_kernel(const EngineMember* __restrict__ table,
                                                                             const long long* __restrict__ prefix,
                                                                             long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        unsigned flags = 0;
        transport_update_cell4<kFp32>(M.T, reinterpret_cast<const float4*>(M.q4), [&](int s) { return engine_scalar(M, s); },
                                      [&](int s) { return engine_scalar_out(M, s); }, M.rho, M.rho_begin,
                                      reinterpret_cast<const float4*>(M.sf), reinterpret_cast<const float4*>(M.rl), c,
                                      flags);
        if (flags) atomicOr(M.status, flags);
    });
}

// The three transport passes with the members' constants in the constant
// bank: a compact copy of each member's transport parameters and its buffers
// that do not rotate; the end-of-loop density and the rain, which rotate,
// are read from the table.
struct TransportConst
{
    TransportCompact T;
    const float4* q4;
    const float *mfx, *mfy, *mfz, *rho_begin;
    float4 *sf, *rl;
    float *theta, *qv, *qc;
    unsigned* status;
};

constexpr int kTransportConstMembers = 64;

struct TransportLaunch
{
    long long prefix[kTransportConstMembers + 1];
    TransportConst m[kTransportConstMembers];
};
static_assert(sizeof(TransportLaunch) <= 32000, "a kernel parameter block holds at most 32764 bytes");

// Calls fn(A, M, c) for every cell of the first tiles of the launch.
template <class Fn>
__device__ __forceinline__ void for_transport_cells(const TransportLaunch& L, const EngineMember* __restrict__ table,
                                                    long long tiles, Fn&& fn)
{
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const TransportConst& A = L.m[m];
        const int c = (int)((t - L.prefix[m]) * blockDim.x) + (int)threadIdx.x;
        if (c >= A.T.d.cells()) continue;
        fn(A, table[m], c);
    }
}

template <bool kFp32>
static __global__ void __launch_bounds__(256, kFp32 ? NIMBUS_FACES_MINB_F32 : NIMBUS_FACES_MINB) engine_transport_faces_const_kernel(
    const __grid_constant__ TransportLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    for_transport_cells(L, table, tiles, [&](const TransportConst& A, const EngineMember&, int c) {
        transport_faces_cell4<kFp32>(A.T, A.q4, A.mfx, A.mfy, A.mfz, A.sf, c);
    });
}

// Of the limiter: the FP32 form at 5 (4 / 5 / 6 / 8: 2.31 / 2.31 / 2.39 / 3.10
// ms), the reference-precision form at 3 (3 / 6 / 8: 0.23 / 0.26 / 0.30).
#ifndef NIMBUS_LIMITER_MINB_F32
#define NIMBUS_LIMITER_MINB_F32 5
#endif
template <bool kFp32>
static __global__ void __launch_bounds__(256, kFp32 ? NIMBUS_LIMITER_MINB_F32 : 3) engine_transport_limiter_const_kernel(
    const __grid_constant__ TransportLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    for_transport_cells(L, table, tiles, [&](const TransportConst& A, const EngineMember&, int c) {
        transport_limiter_cell4<kFp32>(A.T, A.q4, A.rho_begin, A.sf, A.rl, c);
    });
}

// Of the update: both at 3, since the loads of a cell's six faces for four
// scalars are in flight together (FP32 2 / 3 / 4: 3.83 / 3.12 / 3.63 ms;
// reference precision 2 / 3 / 4: 0.42 / 0.35 / 0.41).
#ifndef NIMBUS_UPDATE_MINB_F32
#define NIMBUS_UPDATE_MINB_F32 3
#endif
template <bool kFp32>
static __global__ void __launch_bounds__(256, kFp32 ? NIMBUS_UPDATE_MINB_F32 : 3) engine_transport_update_const_kernel(
    const __grid_constant__ TransportLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    for_transport_cells(L, table, tiles, [&](const TransportConst& A, const EngineMember& M, int c) {
        unsigned flags = 0;
        float* const in_place[4] = {A.theta, A.qv, A.qc, M.qr};
        transport_update_cell4<kFp32>(A.T, A.q4, [&](int s) { return (const float*)in_place[s]; },
                                      [&](int s) { return in_place[s]; }, M.rho, A.rho_begin, A.sf, A.rl, c, flags);
        if (flags) atomicOr(A.status, flags);
    });
}

// ---- Acoustic speed scan before a large step --------------------------------
// Per member the largest (gamma p) / rho of its cells, as ordered double bits
// into c2[row] (row = the member's table row in this launch), for the
// substep count the reference re-derives before every large step
// (src/numerics/runtime.cpp:346-401,854-880).  The member of a tile is
// block-uniform, so a block keeps a running maximum while it walks one
// member's tiles and publishes it with one atomicMax when it moves on.
// One thread reads a group of four cells (one 16-byte load of each field).
static __global__ void __launch_bounds__(kQuadTile) engine_sound_speed_kernel(const EngineMember* __restrict__ table,
                                                                              const long long* __restrict__ prefix,
                                                                              long long tiles, unsigned long long* c2)
{
    grid_dependency();
    int m = 0, held = -1;
    unsigned long long best = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= prefix[m + 1]) ++m;
        if (m != held)
        {
            if (held >= 0)
            {
                const unsigned long long b = block_max_u64(best);
                if (threadIdx.x == 0 && b) atomicMax(c2 + held, b);
            }
            held = m;
            best = 0;
        }
        const EngineMember& M = table[m];
        const int c = 4 * ((int)(t - prefix[m]) * kQuadTile + (int)threadIdx.x);
        if (c >= M.items[kItemCells]) continue;
        unsigned flags = 0;
        int i, j, k;
        decompose(M.F.d, c, i, j, k);
        const Quad p = load_quad(M.p, c), r = load_quad(M.rho, c);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (k + q < M.F.d.nz) best = max(best, sound_speed_sq_bits(M.gamma, p.v[q], r.v[q], flags));
        if (flags) atomicOr(M.status, flags);
    }
    if (held >= 0)
    {
        const unsigned long long b = block_max_u64(best);
        if (threadIdx.x == 0 && b) atomicMax(c2 + held, b);
    }
}

// ---- Kessler and EOS --------------------------------------------------------

// The Kessler step and the EOS re-projection in one pass: the candidate
// pressure is formed from the applied state while it is still in registers
// and written to the member's candidate buffer; engine_swap_kernel publishes
// it by exchanging p and the candidate unless the projection was refused.
// Resident CTAs per SM of the Kessler + EOS pass: the FP32 form at 6 (5 / 6 / 7:
// 4.55 / 4.47 / 4.62 ms), the reference-precision form at 5 (3 / 4 / 5 / 6:
// 0.64 / 0.57 / 0.55 / 0.58).
#ifndef NIMBUS_MICRO_MINB_F32
#define NIMBUS_MICRO_MINB_F32 6
#endif

// A member's constants of the pass, and its buffers that do not rotate.
struct MicroConst
{
    KesslerParams K;
    float *u, *v, *w, *theta, *qv, *qc;
    unsigned* status;
    const float4* eos0;
    EosSeries eos_series;
    double gamma;
    RelaxTables R;
    int microphysics;
};

// The buffers that rotate: density, pressure, rain and its new values, and
// the candidate pressure.
struct MicroRotating
{
    const float *rho, *p, *qr;
    float *qr_alt, *eos;
};

__host__ __device__ __forceinline__ MicroConst micro_const_of(const EngineMember& M)
{
    MicroConst A;
    A.K = M.K;
    A.u = M.u;
    A.v = M.v;
    A.w = M.w;
    A.theta = M.theta;
    A.qv = M.qv;
    A.qc = M.qc;
    A.status = M.status;
    A.eos0 = M.eos0;
    A.eos_series = M.eos_series;
    A.gamma = M.gamma;
    A.R = M.R;
    A.microphysics = M.microphysics;
    return A;
}

template <bool kFp32>
__device__ __forceinline__ void microphysics_eos_cell(const MicroConst& A, const MicroRotating& M, int c)
{
    unsigned flags = 0;
    int i, j, k;
    decompose(A.K.d, c, i, j, k);
    if (k >= A.K.d.nz) return;
    float4 s;
    const float po = M.p[c];
    if (A.microphysics)
    {
        if constexpr (kFp32)
            kessler_cell_f32<true>(A.K, A.theta, A.qv, A.qc, M.qr, M.p, M.rho, M.qr_alt, nullptr, nullptr, nullptr,
                                   nullptr, c, &s);
        else
            kessler_cell<true>(A.K, A.theta, A.qv, A.qc, M.qr, M.p, M.rho, M.qr_alt, nullptr, nullptr, nullptr,
                               nullptr, c, &s);
    }
    else
        s = make_float4(A.theta[c], A.qv[c], A.qc[c], M.qr[c]);
    float p_new;
    bool ok;
    if constexpr (kFp32)
        ok = eos_candidate_value_f32(A.K.d, c, k, M.rho[c], s.x, A.eos0, A.eos_series, A.gamma, true, po, s.y, s.z,
                                     s.w, p_new, flags);
    else
        ok = eos_candidate_value(A.K.d, c, M.rho[c], s.x, A.gamma, true, po, s.y, s.z, s.w, p_new, flags);
    if (ok) M.eos[c] = p_new;
    if (flags) atomicOr(A.status, flags);
    // The end-of-step sponge after the EOS projection (dynamics.cpp:7323-7340).
    if (A.R.do_upper | A.R.do_w_only | A.R.do_lateral)
    {
        float uu = A.u[c], vv = A.v[c], ww = A.w[c], th = s.x;
        if (relax_cell(A.R, A.K.d.nx, A.K.d.ny, i, j, k, uu, vv, ww, th))
        {
            A.u[c] = uu;
            A.v[c] = vv;
            A.w[c] = ww;
            A.theta[c] = th;
        }
    }
}

template <bool kFp32>
static __global__ void __launch_bounds__(256, kFp32 ? NIMBUS_MICRO_MINB_F32 : 5) engine_microphysics_eos_kernel(const EngineMember* __restrict__ table,
                                                                             const long long* __restrict__ prefix,
                                                                             long long tiles)
{
    grid_dependency();
    for_member_items(table, prefix, tiles, kItemCells, [&](const EngineMember& M, int c) {
        microphysics_eos_cell<kFp32>(micro_const_of(M), MicroRotating{M.rho, M.p, M.qr, M.qr_alt, M.eos}, c);
    });
}

// The same with the members' constants in the constant bank, for lanes whose
// constants fit a parameter block: the member table's loads and the registers
// that held them go.  24 members of 16.5 million cells, ten steps 5.45 -> 4.93
// ms; 256x256x80 1.54 -> 1.42; four steps of 3.0 million cells in reference
// precision 0.76 -> 0.73.
constexpr int kMicroConstMembers = 64;

struct MicroLaunch
{
    long long prefix[kMicroConstMembers + 1];
    MicroConst m[kMicroConstMembers];
};
static_assert(sizeof(MicroLaunch) <= 32000, "a kernel parameter block holds at most 32764 bytes");

template <bool kFp32>
static __global__ void __launch_bounds__(256, kFp32 ? NIMBUS_MICRO_MINB_F32 : 5) engine_microphysics_eos_const_kernel(
    const __grid_constant__ MicroLaunch L, const EngineMember* __restrict__ table, long long tiles)
{
    grid_dependency();
    int m = 0;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x)
    {
        while (t >= L.prefix[m + 1]) ++m;
        const MicroConst& A = L.m[m];
        const int c = (int)((t - L.prefix[m]) * blockDim.x) + (int)threadIdx.x;
        if (c >= A.K.d.cells()) continue;
        const EngineMember& M = table[m];
        microphysics_eos_cell<kFp32>(A, MicroRotating{M.rho, M.p, M.qr, M.qr_alt, M.eos}, c);
    }
}

}  // namespace nimbus
