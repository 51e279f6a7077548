// fe_p2g.cu -- particle -> grid transfer (K_p2g).
//
// Reference: PICSimulator::TransferParticles2Grid (pic_simulator.cpp:356-437), FLIPSimulator
// (flip_simulator.cpp:25-119) and APICSimulator (apic_simulator.cpp:15-118): for every particle and
// every velocity component, trilinear weights w on the 8 surrounding faces (GetCooridnatesAndWeights,
// common/math_utils.hpp:75-112), u += w * value, weight += w, marker = 1; then u /= weight where
// weight > 0.  PIC and APIC clamp the face index with the CELL count, FLIP with the face count.  APIC
// adds C_row . (x_face - x_clamped), the particle position clamped by h/2 on the two transverse axes.
//
// B200 design: a block takes a quarter of an 8x8x8-cell tile, one thread per cell.  A tile's particles are one
// contiguous run of the sorted arrays (fe_keys.h) and a cell's particles a contiguous piece of that run, so
// each thread walks its own cell's particles once and sums all three components in registers.  With the domain origin
// at zero the faces a particle of cell (cx, cy, cz) touches lie in a window around the cell -- faces c and c + 1
// along the component's own axis, c - 1 .. c + 1 along the two others -- so a thread's sums live in 18 slots per
// component, (numerator, weight) per window face in one register pair for the packed FMA, plus a touched mask.  The
// block's cells are first put in order of their particle counts, so a warp's lanes walk about equally many.  Only
// then do the threads add their slots into the 10x10x4 face box in shared memory, slot after slot with a barrier
// between: a slot is another face for every cell, so the adds need no atomics (shared FP32 atomics are compare-and-swap
// loops).  Cells with more than kCellCap particles (particles clamped onto a wall pile up in one
// cell) hand the rest to a warp that spreads them over its lanes and combines the lanes' slots by shuffles.
// The box is then flushed to global accumulators: box faces touched by the block get one global red.add each,
// so a face receives a few global adds (one per neighbouring part), never one per particle.  A second pass
// divides numerator by weight and, for FLIP, writes the snapshot (flip_simulator.cpp:107-118).  A particle
// whose stencil leaves its cell's window (only possible for a domain origin away from zero, where the
// reference's data origins ignore the origin) takes the direct path instead: shared atomics into the box per
// face, or global adds for faces outside the box, so the kernel stays correct for every input.
//
// Bound by instruction issue and the latency of a walk at 3 blocks (APIC 2) per SM.  A whole tile per block with one walk
// per component and atomic box adds against this, the stage with its clears and normalisation: 65 against 60 us at 32^3
// FLIP, 100 against 83 at 64^3 PIC, 138 against 106 at 61x90x47 APIC, 342 against 231 at 128^3 FLIP (4 M particles; the
// splat kernels alone 249 against 176), 489 against 390 at 128^3 APIC, 1616 against 1326 at 200^3 APIC.
#include <algorithm>

#include "fe_internal.cuh"

namespace fe {
namespace {

// A block takes a quarter of a tile, two cell layers along z, one thread per cell.
constexpr int kP2gLayers = 2, kP2gParts = FE_TILE / kP2gLayers;
constexpr int kP2gThreads = FE_TILE * FE_TILE * kP2gLayers;
constexpr int kBox = 10, kBoxZ = kP2gLayers + 2;  // faces of the part and one around it
constexpr int kBoxFaces = kBox * kBox * kBoxZ;
constexpr int kCellCap = 32;                // particles a thread sums for its own cell; the rest go to a warp

// Per-component constants of the transfer (face-array sizes, the clamp sizes the reference passes to
// GetCooridnatesAndWeights, the data origin, the global accumulators).
struct P2gComp {
    int fsx, fsy, fsz;  // face-array sizes
    int csx, csy, csz;  // clamp sizes: FLIP the face counts, PIC / APIC the cell counts
    float org[3];       // data origin of the component's face grid
    float* gnum;
    float* gden;
    uint8_t* gmk;
};

template <int SOLVER>
__device__ __forceinline__ P2gComp p2g_comp(const SceneView& v, int c)
{
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const bool flip = SOLVER == FE_SOLVER_FLIP;
    P2gComp k;
    k.fsx = nx + (c == 0);
    k.fsy = ny + (c == 1);
    k.fsz = nz + (c == 2);
    k.csx = flip ? k.fsx : nx;
    k.csy = flip ? k.fsy : ny;
    k.csz = flip ? k.fsz : nz;
#pragma unroll
    for (int a = 0; a < 3; ++a) k.org[a] = c == 0 ? v.xo[a] : (c == 1 ? v.yo[a] : v.zo[a]);
    k.gnum = c == 0 ? v.nu : (c == 1 ? v.nv : v.nw);
    k.gden = c == 0 ? v.du : (c == 1 ? v.dv : v.dw);
    k.gmk = c == 0 ? v.mu : (c == 1 ? v.mv : v.mw);
    return k;
}

// A particle's value for component c and its (APIC) clamped position and C row.
template <int SOLVER>
struct P2gParticle {
    float vc;
    float pc[3];
    float cr[3];
};

template <int SOLVER>
__device__ __forceinline__ P2gParticle<SOLVER> load_particle(const SceneView& v, uint32_t p, int c, float x, float y,
                                                             float z, const float lo[3], const float hi[3])
{
    P2gParticle<SOLVER> q;
    q.vc = __ldg((c == 0 ? v.vx : (c == 1 ? v.vy : v.vz)) + p);
    q.pc[0] = x;
    q.pc[1] = y;
    q.pc[2] = z;
    q.cr[0] = q.cr[1] = q.cr[2] = 0.f;
    if (SOLVER == FE_SOLVER_APIC) {
        q.cr[0] = __ldg(v.c[3 * c] + p);
        q.cr[1] = __ldg(v.c[3 * c + 1] + p);
        q.cr[2] = __ldg(v.c[3 * c + 2] + p);
        // Clamp(val, max, min) on the two transverse axes (apic_simulator.cpp:55-57,68-70,81-83)
#pragma unroll
        for (int a = 0; a < 3; ++a)
            if (a != c) q.pc[a] = q.pc[a] < lo[a] ? lo[a] : (q.pc[a] > hi[a] ? hi[a] : q.pc[a]);
    }
    return q;
}

// The particle's 8 faces added one by one: into the box (shared atomics) or, outside it, into the global
// accumulators.  Used for particles whose stencil leaves their cell's window.
template <int SOLVER>
__device__ __forceinline__ void splat_direct(const SceneView& v, const P2gComp& k, const Stencil& s, const P2gParticle<SOLVER>& q,
                             int bx, int by, int bz, float* s_num, float* s_den, uint8_t* s_mk)
{
    const float wx[2] = {1.f - s.fx, s.fx}, wy[2] = {1.f - s.fy, s.fy}, wz[2] = {1.f - s.fz, s.fz};
    const int ii[2] = {s.i, s.ip}, jj[2] = {s.j, s.jp}, kk[2] = {s.k, s.kp};
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int a = t & 1, b = (t >> 1) & 1, d = t >> 2;
        const float wgt = wx[a] * wy[b] * wz[d];
        float val = q.vc;
        if (SOLVER == FE_SOLVER_APIC) {
            const float gx = k.org[0] + v.hf[0] * (float)ii[a];
            const float gy = k.org[1] + v.hf[1] * (float)jj[b];
            const float gz = k.org[2] + v.hf[2] * (float)kk[d];
            val += q.cr[0] * (gx - q.pc[0]) + q.cr[1] * (gy - q.pc[1]) + q.cr[2] * (gz - q.pc[2]);
        }
        const int li = ii[a] - bx, lj = jj[b] - by, lk = kk[d] - bz;
        if ((unsigned)li < kBox && (unsigned)lj < kBox && (unsigned)lk < kBoxZ) {
            const int l = li + kBox * (lj + kBox * lk);
            atomicAdd(&s_num[l], val * wgt);
            atomicAdd(&s_den[l], wgt);
            s_mk[l] = 1;
        } else {
            const size_t f = idx3(ii[a], jj[b], kk[d], k.fsx, k.fsy);
            atomicAdd(k.gnum + f, val * wgt);
            atomicAdd(k.gden + f, wgt);
            k.gmk[f] = 1;
        }
    }
}

// Window of component C's faces around a cell: along the component's own (staggered) axis a particle of cell c
// touches faces c and c + 1, along the two other axes c - 1 .. c + 1.  Slot (i, j, k) of the window is face
// (cx + lo<C>(0) + i, cy + lo<C>(1) + j, cz + lo<C>(2) + k), slot index i + W0 (j + W1 k).
template <int C> __host__ __device__ constexpr int win(int axis) { return axis == C ? 2 : 3; }
template <int C> __host__ __device__ constexpr int wlo(int axis) { return axis == C ? 0 : -1; }
template <int C> __host__ __device__ constexpr int nslots() { return win<C>(0) * win<C>(1) * win<C>(2); }  // 18
// `count` ones spaced `width` bits apart (bit 0, width, 2 width, ...).
__host__ __device__ constexpr uint32_t rep_bits(int width, int count)
{
    return count <= 0 ? 0u : (rep_bits(width, count - 1) << width) | 1u;
}

// Touched slots of the window from each axis' touched bits (tx over W0, ty over W1, tz over W2): slot (a, b, c)
// is touched when bit a of tx, b of ty and c of tz are, found by spreading each axis' bits over the slot layout.
template <int C>
__host__ __device__ constexpr uint32_t spread_mask(uint32_t tx, uint32_t ty, uint32_t tz)
{
    constexpr int W0 = win<C>(0), W1 = win<C>(1), W2 = win<C>(2);
    uint32_t sy = 0, ez = 0;
    for (int b3 = 0; b3 < W1; ++b3) sy |= ((ty >> b3) & 1u) * (((1u << W0) - 1u) << (W0 * b3));
    for (int c3 = 0; c3 < W2; ++c3) ez |= ((tz >> c3) & 1u) * (((1u << (W0 * W1)) - 1u) << (W0 * W1 * c3));
    return (tx * rep_bits(W0, W1 * W2)) & (sy * rep_bits(W0 * W1, W2)) & ez;
}
// Touched slots of an unclamped particle in the lower half of the cell on every transverse axis (the first two
// faces of each axis); the upper halves shift it by one face per axis.
template <int C>
__host__ __device__ constexpr uint32_t regular_mask()
{
    return spread_mask<C>(3u, 3u, 3u);
}

// One particle of cell (cx, cy, cz) into the cell's 18 slots of component C; returns false (and adds nothing)
// when its stencil leaves the window, in which case the caller takes the direct path.  The trilinear weight of
// slot (i, j, k) is wx_i wy_j wz_k, so the sums are formed as wx_i (wy_j wz_k v) per (j, k) pair: 2 FMAs per slot
// (APIC: v + C . (x_face - x_p) splits the same way, 3 FMAs per slot).
template <int SOLVER, int C>
__device__ __forceinline__ bool splat_slots(const SceneView& v, const P2gComp& k, const Stencil& s,
                                            const P2gParticle<SOLVER>& q, int cx, int cy, int cz,
                                            float (&num)[nslots<C>()], float (&den)[nslots<C>()], uint32_t& mask)
{
    constexpr int W0 = win<C>(0), W1 = win<C>(1), W2 = win<C>(2);
    constexpr int L0 = wlo<C>(0), L1 = wlo<C>(1), L2 = wlo<C>(2);
    const int oi = s.i - cx, oip = s.ip - cx, oj = s.j - cy, ojp = s.jp - cy, ok = s.k - cz, okp = s.kp - cz;
    if (oi < L0 || oip > L0 + W0 - 1 || oj < L1 || ojp > L1 + W1 - 1 || ok < L2 || okp > L2 + W2 - 1) return false;
    float wx[W0], wy[W1], wz[W2];
    // The usual case: no clamp on any axis, so the stencil is the cell's two own-axis faces and, on each transverse
    // axis, the lower or the upper two of the window's three faces (the half of the cell the particle is in).  The
    // weights are then selects of (1 - f, f), the same values the general sums below give, and the touched slots a
    // fixed pattern shifted by those halves.
    auto axis_regular = [](int o, int op, int W, int lo) { return op == o + 1 && (o == lo || (W == 3 && o == lo + 1)); };
    const bool regular = axis_regular(oi, oip, W0, L0) && axis_regular(oj, ojp, W1, L1) && axis_regular(ok, okp, W2, L2);
    if (regular) {
        const bool hx = W0 == 3 && oi == L0 + 1;
        const bool hy = W1 == 3 && oj == L1 + 1;
        const bool hz = W2 == 3 && ok == L2 + 1;
        const float f[3] = {s.fx, s.fy, s.fz};
        const bool h[3] = {hx, hy, hz};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int W = a == 0 ? W0 : (a == 1 ? W1 : W2);
            float* w = a == 0 ? wx : (a == 1 ? wy : wz);
            const float lo = 1.f - f[a];
            if (W == 2) {
                w[0] = lo;
                w[1] = f[a];
            } else {
                w[0] = h[a] ? 0.f : lo;
                w[1] = h[a] ? lo : f[a];
                w[2 % W] = h[a] ? f[a] : 0.f;
            }
        }
        mask |= regular_mask<C>() << ((hx ? 1 : 0) + W0 * ((hy ? 1 : 0) + W1 * (hz ? 1 : 0)));
    } else {
        // 1D weights and touched bits on the window (i and ip coincide only on a one-face axis)
        uint32_t tx = 0, ty = 0, tz = 0;
#pragma unroll
        for (int r = 0; r < W0; ++r) {
            wx[r] = (oi == L0 + r ? 1.f - s.fx : 0.f) + (oip == L0 + r ? s.fx : 0.f);
            tx |= (oi == L0 + r || oip == L0 + r) ? 1u << r : 0u;
        }
#pragma unroll
        for (int r = 0; r < W1; ++r) {
            wy[r] = (oj == L1 + r ? 1.f - s.fy : 0.f) + (ojp == L1 + r ? s.fy : 0.f);
            ty |= (oj == L1 + r || ojp == L1 + r) ? 1u << r : 0u;
        }
#pragma unroll
        for (int r = 0; r < W2; ++r) {
            wz[r] = (ok == L2 + r ? 1.f - s.fz : 0.f) + (okp == L2 + r ? s.fz : 0.f);
            tz |= (ok == L2 + r || okp == L2 + r) ? 1u << r : 0u;
        }
        mask |= spread_mask<C>(tx, ty, tz);
    }
    float gx[W0];  // APIC: wx_i C_x (x_face_i - x_p)
    float dy[W1], dz[W2];
    if (SOLVER == FE_SOLVER_APIC) {
#pragma unroll
        for (int r = 0; r < W0; ++r) gx[r] = wx[r] * (q.cr[0] * ((k.org[0] + v.hf[0] * (float)(cx + L0 + r)) - q.pc[0]));
#pragma unroll
        for (int r = 0; r < W1; ++r) dy[r] = (k.org[1] + v.hf[1] * (float)(cy + L1 + r)) - q.pc[1];
#pragma unroll
        for (int r = 0; r < W2; ++r) dz[r] = (k.org[2] + v.hf[2] * (float)(cz + L2 + r)) - q.pc[2];
    }
#pragma unroll
    for (int c3 = 0; c3 < W2; ++c3)
#pragma unroll
        for (int b3 = 0; b3 < W1; ++b3) {
            const float a = wy[b3] * wz[c3];
            float val = q.vc;
            if (SOLVER == FE_SOLVER_APIC) val += q.cr[1] * dy[b3] + q.cr[2] * dz[c3];
            const float t = a * val;
#pragma unroll
            for (int a3 = 0; a3 < W0; ++a3) {
                const int slot = a3 + W0 * (b3 + W1 * c3);
                if (SOLVER == FE_SOLVER_APIC) num[slot] += wx[a3] * t + gx[a3] * a;
                else num[slot] += wx[a3] * t;
                den[slot] += wx[a3] * a;
            }
        }
    return true;
}

// Box index of slot `slot` of component C for the cell at tile-local (lx, ly, lz): the box starts one face before
// the tile.
template <int C>
__device__ __forceinline__ int slot_box(int lx, int ly, int lz, int slot)
{
    constexpr int W0 = win<C>(0), W1 = win<C>(1);
    const int a = slot % W0, b = (slot / W0) % W1, c = slot / (W0 * W1);
    return (lx + 1 + wlo<C>(0) + a) + kBox * ((ly + 1 + wlo<C>(1) + b) + kBox * (lz + 1 + wlo<C>(2) + c));
}

// Component C of the cell's particles [pb, pe) (a thread's own cell, or a warp's share of a crowded cell with
// lane stride 32) into the slots.
template <int SOLVER, int C>
__device__ __forceinline__ void cell_component(const SceneView& v, uint32_t pb, uint32_t pe, uint32_t stride, int cx,
                                               int cy, int cz, int bx, int by, int bz, const float lo[3],
                                               const float hi[3], float (&num)[nslots<C>()],
                                               float (&den)[nslots<C>()], uint32_t& mask, float* s_num, float* s_den,
                                               uint8_t* s_mk)
{
    const P2gComp k = p2g_comp<SOLVER>(v, C);
#pragma unroll
    for (int t = 0; t < nslots<C>(); ++t) num[t] = den[t] = 0.f;
    mask = 0;
    for (uint32_t p = pb; p < pe; p += stride) {
        const float x = __ldg(v.px + p), y = __ldg(v.py + p), z = __ldg(v.pz + p);  // read-only during P2G
        const Stencil s = stencil(x, y, z, k.org, v.inv_hf, k.csx, k.csy, k.csz);
        const P2gParticle<SOLVER> q = load_particle<SOLVER>(v, p, C, x, y, z, lo, hi);
        if (!splat_slots<SOLVER, C>(v, k, s, q, cx, cy, cz, num, den, mask))
            splat_direct<SOLVER>(v, k, s, q, bx, by, bz, s_num, s_den, s_mk);
    }
}

template <int SOLVER, int C>
__device__ __forceinline__ void flush_slots(int lx, int ly, int lz, const float (&num)[nslots<C>()],
                                            const float (&den)[nslots<C>()], uint32_t mask, float* s_num, float* s_den,
                                            uint8_t* s_mk)
{
#pragma unroll
    for (int t = 0; t < nslots<C>(); ++t) {
        if (!((mask >> t) & 1u)) continue;
        const int l = slot_box<C>(lx, ly, lz, t);
        atomicAdd(&s_num[l], num[t]);
        atomicAdd(&s_den[l], den[t]);
        s_mk[l] = 1;
    }
}

// A crowded cell's particles past kCellCap, spread over a warp's lanes; the lanes' slots are summed by shuffles
// and lane 0 adds them into the box.
template <int SOLVER, int C>
__device__ __forceinline__ void crowded_component(const SceneView& v, uint32_t ob, uint32_t oe, int ox, int oy, int oz,
                                                  int cx, int cy, int cz, int bx, int by, int bz, const float lo[3],
                                                  const float hi[3], float* s_num, float* s_den, uint8_t* s_mk)
{
    const int lane = threadIdx.x & 31;
    float num[nslots<C>()], den[nslots<C>()];
    uint32_t mask;
    cell_component<SOLVER, C>(v, ob + lane, oe, 32u, cx, cy, cz, bx, by, bz, lo, hi, num, den, mask, s_num, s_den,
                              s_mk);
    mask = __reduce_or_sync(0xffffffffu, mask);
#pragma unroll
    for (int q = 0; q < nslots<C>(); ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            num[q] += __shfl_xor_sync(0xffffffffu, num[q], off);
            den[q] += __shfl_xor_sync(0xffffffffu, den[q], off);
        }
    if (lane == 0) flush_slots<SOLVER, C>(ox, oy, oz, num, den, mask, s_num, s_den, s_mk);
}

// One axis of a particle's stencils.  The grid staggered along the axis has its two faces at the cell's sides (own
// weights); the two grids that are not share one index and fraction (their data origins and sizes along it are the
// same), the lower or the upper two of the window's three faces.  own_ok / tr_ok: the faces lie in the window.
struct P2gAxis {
    int oi, ti;        // first face of either pair
    float of, tf;      // fractions
    float own[2], tr[3];
    bool own_ok, tr_ok, upper;
    bool last;         // the cell counts clamp the own pair of the last cell's particles to faces c - 1 and c, weights 0, 1
};
__device__ __forceinline__ P2gAxis p2g_axis(float x, float own_org, float tr_org, float ih, int own_size, int n, int c)
{
    P2gAxis a;
    bary((x - own_org) * ih, own_size - 1, a.oi, a.of);
    bary((x - tr_org) * ih, n - 1, a.ti, a.tf);
    a.last = a.oi == c - 1 && a.of == 1.f;
    a.own_ok = a.oi == c || a.last;
    a.upper = a.ti == c;
    a.tr_ok = a.upper || a.ti == c - 1;
    a.own[0] = a.last ? 1.f : 1.f - a.of;
    a.own[1] = a.last ? 0.f : a.of;
    const float lo = 1.f - a.tf;
    a.tr[0] = a.upper ? 0.f : lo;
    a.tr[1] = a.upper ? lo : a.tf;
    a.tr[2] = a.upper ? a.tf : 0.f;
    return a;
}

// (numerator, weight) of a face in one 64-bit register pair: the packed FP32 FMA adds to both at once.
using Sum2 = unsigned long long;
__device__ __forceinline__ Sum2 pack2(float a, float b)
{
    Sum2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(Sum2 s)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(s));
    return r;
}
__device__ __forceinline__ Sum2 fma2(Sum2 a, Sum2 b, Sum2 c)
{
    Sum2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Component C of one particle into the cell's slots from its axes' weights: the sums of splat_slots.
template <int SOLVER, int C>
__device__ __forceinline__ void add_slots(const SceneView& v, const P2gAxis (&ax)[3], const float org[3], float vc,
                                          const float cr[3], const float pc[3], const int c[3], const int l[3],
                                          Sum2 (&sum)[nslots<C>()], uint32_t& mask, uint8_t* s_mk)
{
    constexpr int W0 = win<C>(0), W1 = win<C>(1), W2 = win<C>(2);
    const float* wx = C == 0 ? ax[0].own : ax[0].tr;
    const float* wy = C == 1 ? ax[1].own : ax[1].tr;
    const float* wz = C == 2 ? ax[2].own : ax[2].tr;
    const int up[3] = {C != 0 && ax[0].upper ? 1 : 0, C != 1 && ax[1].upper ? 1 : 0, C != 2 && ax[2].upper ? 1 : 0};
    if (ax[C].last) {  // face c only; face c - 1 is touched with weight 0, which the marks show
        mask |= spread_mask<C>(C == 0 ? 1u : 3u, C == 1 ? 1u : 3u, C == 2 ? 1u : 3u) << (up[0] + W0 * (up[1] + W1 * up[2]));
        const int f[3] = {l[0] + (C == 0 ? 0 : up[0]), l[1] + (C == 1 ? 0 : up[1]), l[2] + (C == 2 ? 0 : up[2])};
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // the other axes' two faces each
            const int g[3] = {f[0] + (C == 0 ? 0 : (q & 1)), f[1] + (C == 1 ? 0 : (C == 0 ? (q & 1) : (q >> 1))),
                              f[2] + (C == 2 ? 0 : (q >> 1))};
            s_mk[g[0] + kBox * (g[1] + kBox * g[2])] = 1;
        }
    } else {
        mask |= regular_mask<C>() << (up[0] + W0 * (up[1] + W1 * up[2]));
    }
    float gx[W0], dy[W1], dz[W2];
    if (SOLVER == FE_SOLVER_APIC) {
#pragma unroll
        for (int r = 0; r < W0; ++r) gx[r] = cr[0] * ((org[0] + v.hf[0] * (float)(c[0] + wlo<C>(0) + r)) - pc[0]);
#pragma unroll
        for (int r = 0; r < W1; ++r) dy[r] = (org[1] + v.hf[1] * (float)(c[1] + wlo<C>(1) + r)) - pc[1];
#pragma unroll
        for (int r = 0; r < W2; ++r) dz[r] = (org[2] + v.hf[2] * (float)(c[2] + wlo<C>(2) + r)) - pc[2];
    }
    Sum2 w2[W0];
#pragma unroll
    for (int r = 0; r < W0; ++r) w2[r] = pack2(wx[r], wx[r]);
#pragma unroll
    for (int c3 = 0; c3 < W2; ++c3)
#pragma unroll
        for (int b3 = 0; b3 < W1; ++b3) {
            const float a = wy[b3] * wz[c3];
            if (SOLVER == FE_SOLVER_APIC) {
                const float val = vc + (cr[1] * dy[b3] + cr[2] * dz[c3]);
#pragma unroll
                for (int a3 = 0; a3 < W0; ++a3) {
                    Sum2& s = sum[a3 + W0 * (b3 + W1 * c3)];
                    s = fma2(w2[a3], pack2(a * (val + gx[a3]), a), s);
                }
            } else {
                const Sum2 ta = pack2(a * vc, a);
#pragma unroll
                for (int a3 = 0; a3 < W0; ++a3) {
                    Sum2& s = sum[a3 + W0 * (b3 + W1 * c3)];
                    s = fma2(w2[a3], ta, s);
                }
            }
        }
}

// The tile's face box in shared memory (declared by the kernels, so a kernel that runs several transfer kinds holds
// one box, not one per kind).
struct __align__(16) P2gShared {
    float num[3][kBoxFaces];
    float den[3][kBoxFaces];
    uint8_t mk[3][kBoxFaces];
    uint16_t over[kP2gThreads];    // cells with more than kCellCap particles (index in the part)
    int nover;
    int bin[kCellCap + 1];
    uint16_t order[kP2gThreads];
};
static_assert(kCellCap == 32, "one lane per count below the cap");

// Slot t of the window is another face for every cell, so the block adds slot after slot with a barrier between instead of
// atomically (shared FP32 atomics are compare-and-swap loops).
template <int C>
__device__ __forceinline__ void flush_slot(int t, const int l[3], Sum2 sum, uint32_t mask, P2gShared& sh)
{
    if ((mask >> t) & 1u) {
        const int f = slot_box<C>(l[0], l[1], l[2], t);
        const float2 s = unpack2(sum);
        sh.num[C][f] += s.x;
        sh.den[C][f] += s.y;
        sh.mk[C][f] = 1;
    }
}

// A component of a particle whose faces leave the window (a domain origin away from zero).
template <int SOLVER, int C>
__device__ __forceinline__ void add_direct(const SceneView& v, uint32_t p, int bx, int by, int bz, const float lo[3],
                                        const float hi[3], float* s_num, float* s_den, uint8_t* s_mk)
{
    const P2gComp k = p2g_comp<SOLVER>(v, C);
    const float x = __ldg(v.px + p), y = __ldg(v.py + p), z = __ldg(v.pz + p);
    const Stencil s = stencil(x, y, z, k.org, v.inv_hf, k.csx, k.csy, k.csz);
    splat_direct<SOLVER>(v, k, s, load_particle<SOLVER>(v, p, C, x, y, z, lo, hi), bx, by, bz, s_num, s_den, s_mk);
}


// The cell's particles [pb, pe), all three components in one walk: 108 sums in registers, a particle's position and
// velocity read once and its six axis weights computed once (three walks, one per component: 1224 thread instructions a
// particle at 64^3 FLIP).
template <int SOLVER>
__device__ __forceinline__ void own_cell(const SceneView& v, uint32_t pb, uint32_t pe, const int c[3], const int l[3],
                                         int bx, int by, int bz, const float lo[3], const float hi[3], P2gShared& sh)
{
    const bool flip = SOLVER == FE_SOLVER_FLIP;
    Sum2 s0[18], s1[18], s2[18];
#pragma unroll
    for (int t = 0; t < 18; ++t) s0[t] = s1[t] = s2[t] = 0ull;
    uint32_t m0 = 0, m1 = 0, m2 = 0;
    for (uint32_t p = pb; p < pe; ++p) {
        const float X[3] = {__ldg(v.px + p), __ldg(v.py + p), __ldg(v.pz + p)};
        const float V[3] = {__ldg(v.vx + p), __ldg(v.vy + p), __ldg(v.vz + p)};
        float cr[9], q[3] = {0.f, 0.f, 0.f};
        if (SOLVER == FE_SOLVER_APIC) {
#pragma unroll
            for (int k = 0; k < 9; ++k) cr[k] = __ldg(v.c[k] + p);
            // Clamp(val, max, min) on the transverse axes (apic_simulator.cpp:55-57,68-70,81-83)
#pragma unroll
            for (int a = 0; a < 3; ++a) q[a] = X[a] < lo[a] ? lo[a] : (X[a] > hi[a] ? hi[a] : X[a]);
        } else {
#pragma unroll
            for (int k = 0; k < 9; ++k) cr[k] = 0.f;
        }
        const P2gAxis ax[3] = {p2g_axis(X[0], v.xo[0], v.yo[0], v.inv_hf[0], flip ? v.g.nx + 1 : v.g.nx, v.g.nx, c[0]),
                               p2g_axis(X[1], v.yo[1], v.xo[1], v.inv_hf[1], flip ? v.g.ny + 1 : v.g.ny, v.g.ny, c[1]),
                               p2g_axis(X[2], v.zo[2], v.xo[2], v.inv_hf[2], flip ? v.g.nz + 1 : v.g.nz, v.g.nz, c[2])};
        const float pu[3] = {X[0], q[1], q[2]}, pv[3] = {q[0], X[1], q[2]}, pw[3] = {q[0], q[1], X[2]};
        if (ax[0].own_ok && ax[1].tr_ok && ax[2].tr_ok) add_slots<SOLVER, 0>(v, ax, v.xo, V[0], cr, pu, c, l, s0, m0, sh.mk[0]);
        else add_direct<SOLVER, 0>(v, p, bx, by, bz, lo, hi, sh.num[0], sh.den[0], sh.mk[0]);
        if (ax[0].tr_ok && ax[1].own_ok && ax[2].tr_ok) add_slots<SOLVER, 1>(v, ax, v.yo, V[1], cr + 3, pv, c, l, s1, m1, sh.mk[1]);
        else add_direct<SOLVER, 1>(v, p, bx, by, bz, lo, hi, sh.num[1], sh.den[1], sh.mk[1]);
        if (ax[0].tr_ok && ax[1].tr_ok && ax[2].own_ok) add_slots<SOLVER, 2>(v, ax, v.zo, V[2], cr + 6, pw, c, l, s2, m2, sh.mk[2]);
        else add_direct<SOLVER, 2>(v, p, bx, by, bz, lo, hi, sh.num[2], sh.den[2], sh.mk[2]);
    }
    __syncthreads();  // the direct adds above are atomic and go to the same box
#pragma unroll
    for (int t = 0; t < 18; ++t) {
        flush_slot<0>(t, l, s0[t], m0, sh);
        flush_slot<1>(t, l, s1[t], m1, sh);
        flush_slot<2>(t, l, s2[t], m2, sh);
        __syncthreads();
    }
}

// Parts of at most kFewParticles particles (spray) add each particle's faces to the global accumulators: setting up and
// flushing the box would cost more.  `first` of `step` threads.
constexpr uint32_t kFewParticles = 32;
template <int SOLVER>
__device__ __forceinline__ void few_particles(const SceneView& v, uint32_t beg, uint32_t end, uint32_t first, uint32_t step)
{
    const float lo[3] = {v.originf[0] + 0.5f * v.hf[0], v.originf[1] + 0.5f * v.hf[1], v.originf[2] + 0.5f * v.hf[2]};
    const float hi[3] = {v.originf[0] + v.sizef[0] - 0.5f * v.hf[0], v.originf[1] + v.sizef[1] - 0.5f * v.hf[1],
                         v.originf[2] + v.sizef[2] - 0.5f * v.hf[2]};
    for (uint32_t e = first; e < 3 * (end - beg); e += step) {
        const uint32_t p = beg + e / 3;
        const int c = (int)(e % 3);
        const P2gComp k = p2g_comp<SOLVER>(v, c);
        const float x = __ldg(v.px + p), y = __ldg(v.py + p), z = __ldg(v.pz + p);
        const Stencil s = stencil(x, y, z, k.org, v.inv_hf, k.csx, k.csy, k.csz);
        // a box that no face lies in: every face goes to the global accumulators
        splat_direct<SOLVER>(v, k, s, load_particle<SOLVER>(v, p, c, x, y, z, lo, hi), 1 << 24, 1 << 24, 1 << 24, nullptr,
                             nullptr, nullptr);
    }
}
__device__ __forceinline__ uint32_t part_first_key(int part)
{
    return (uint32_t)(part / kP2gParts) * FE_TILE_CELLS + (uint32_t)(part % kP2gParts) * (uint32_t)kP2gThreads;
}

// A warp per part: parts of few particles are done here, at full occupancy; the others are listed for k_p2g, whose blocks
// (168 registers a thread) would otherwise mostly start up for parts with nothing or little to do.
template <int SOLVER>
__global__ void __launch_bounds__(256) k_p2g_few(SceneView v, int parts)
{
    const int part = (int)(blockIdx.x * 8 + (threadIdx.x >> 5)), lane = (int)(threadIdx.x & 31);
    if (part >= parts) return;
    const uint32_t first = part_first_key(part);
    const uint32_t beg = v.cell_start[first], end = v.cell_start[first + kP2gThreads];
    if (end - beg > kFewParticles) {
        if (lane == 0) v.p2g_list[2 + atomicAdd(v.p2g_list, 1u)] = (uint32_t)part;
    } else {
        few_particles<SOLVER>(v, beg, end, (uint32_t)lane, 32u);
    }
}

template <int SOLVER>
__device__ __forceinline__ void p2g_body(const SceneView& v, int part, P2gShared& sh)
{
    float (&s_num)[3][kBoxFaces] = sh.num;
    float (&s_den)[3][kBoxFaces] = sh.den;
    uint8_t (&s_mk)[3][kBoxFaces] = sh.mk;
    uint16_t* s_over = sh.over;
    int& s_nover = sh.nover;

    const int tile = part / kP2gParts, layer = part % kP2gParts * kP2gLayers;
    const int tx = tile % v.g.tnx, ty = (tile / v.g.tnx) % v.g.tny, tz = tile / (v.g.tnx * v.g.tny);
    const int x0 = tx * FE_TILE, y0 = ty * FE_TILE, z0 = tz * FE_TILE + layer;
    const int bx = x0 - 1, by = y0 - 1, bz = z0 - 1;  // box origin (face index)
    const uint32_t first = part_first_key(part);
    const uint32_t beg = v.cell_start[first], end = v.cell_start[first + kP2gThreads];
    if (beg == end) return;  // nothing to splat; accumulators were cleared by the caller
    const float lo[3] = {v.originf[0] + 0.5f * v.hf[0], v.originf[1] + 0.5f * v.hf[1], v.originf[2] + 0.5f * v.hf[2]};
    const float hi[3] = {v.originf[0] + v.sizef[0] - 0.5f * v.hf[0], v.originf[1] + v.sizef[1] - 0.5f * v.hf[1],
                         v.originf[2] + v.sizef[2] - 0.5f * v.hf[2]};
    if (end - beg <= kFewParticles) {  // (in a flat batch launch; k_p2g_few has done them otherwise)
        few_particles<SOLVER>(v, beg, end, threadIdx.x, blockDim.x);
        return;
    }

    for (int t = threadIdx.x; t < 3 * kBoxFaces / 4; t += blockDim.x) {
        reinterpret_cast<float4*>(&s_num[0][0])[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<float4*>(&s_den[0][0])[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<uint32_t*>(&s_mk[0][0])[t] = 0u;
    }
    if (threadIdx.x == 0) s_nover = 0;
    if (threadIdx.x <= (unsigned)kCellCap) sh.bin[threadIdx.x] = 0;
    __syncthreads();

    // the part's cells in order of their particle counts, one per thread: a warp's lanes then walk about equally many
    // (in cell order a warp went on until its fullest cell was done: 14 rounds for 8 particles a cell)
    int cell = (int)threadIdx.x;
    {
        const uint32_t count = min(v.cell_start[first + cell + 1] - v.cell_start[first + cell], (uint32_t)kCellCap);
        const int at = atomicAdd(&sh.bin[count], 1);
        __syncthreads();
        if (threadIdx.x < 32) {
            int x = sh.bin[threadIdx.x];
            const int own = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if ((int)threadIdx.x >= o) x += y;
            }
            sh.bin[threadIdx.x] = x - own;
            if (threadIdx.x == 31) sh.bin[kCellCap] = x;
        }
        __syncthreads();
        sh.order[sh.bin[count] + at] = (uint16_t)cell;
        __syncthreads();
        cell = sh.order[threadIdx.x];
    }
    const int l[3] = {cell & 7, (cell >> 3) & 7, cell >> 6};
    const int c[3] = {x0 + l[0], y0 + l[1], z0 + l[2]};
    uint32_t pb = v.cell_start[first + cell], pe = v.cell_start[first + cell + 1];  // none in cells outside the grid
    if (pe - pb > (uint32_t)kCellCap) {
        s_over[atomicAdd(&s_nover, 1)] = (uint16_t)cell;
        pe = pb + kCellCap;
    }
    own_cell<SOLVER>(v, pb, pe, c, l, bx, by, bz, lo, hi, sh);

    // crowded cells: a warp per cell, lanes stride over the particles past kCellCap
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nover = s_nover;
    for (int o = warp; o < nover; o += nwarps) {
        const int t = s_over[o];
        const int ox = t & 7, oy = (t >> 3) & 7, oz = t >> 6;
        const uint32_t ob = v.cell_start[first + (uint32_t)t] + kCellCap, oe = v.cell_start[first + (uint32_t)t + 1];
        crowded_component<SOLVER, 0>(v, ob, oe, ox, oy, oz, x0 + ox, y0 + oy, z0 + oz, bx, by, bz, lo, hi, s_num[0], s_den[0],
                                     s_mk[0]);
        crowded_component<SOLVER, 1>(v, ob, oe, ox, oy, oz, x0 + ox, y0 + oy, z0 + oz, bx, by, bz, lo, hi, s_num[1], s_den[1],
                                     s_mk[1]);
        crowded_component<SOLVER, 2>(v, ob, oe, ox, oy, oz, x0 + ox, y0 + oy, z0 + oz, bx, by, bz, lo, hi, s_num[2], s_den[2],
                                     s_mk[2]);
    }
    __syncthreads();

#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const P2gComp k = p2g_comp<SOLVER>(v, c);
        for (int l = threadIdx.x; l < kBoxFaces; l += blockDim.x) {
            if (!s_mk[c][l]) continue;
            const int li = l % kBox, lj = (l / kBox) % kBox, lk = l / (kBox * kBox);
            const int gi = bx + li, gj = by + lj, gk = bz + lk;
            if (gi < 0 || gj < 0 || gk < 0 || gi >= k.fsx || gj >= k.fsy || gk >= k.fsz) continue;
            const size_t f = idx3(gi, gj, gk, k.fsx, k.fsy);
            atomicAdd(k.gnum + f, s_num[c][l]);
            atomicAdd(k.gden + f, s_den[c][l]);
            k.gmk[f] = 1;
        }
    }
}

template <int SOLVER>
__global__ void __launch_bounds__(kP2gThreads, SOLVER == FE_SOLVER_APIC ? 2 : 3) k_p2g(SceneView v)
{
    __shared__ P2gShared sh;
    __shared__ uint32_t part;
    const uint32_t n = v.p2g_list[0];
    // parts as the blocks get free: one with crowded cells takes many times as long as another.  The next one is asked for
    // before the present one is worked on.  (In turn, the stage took 447 us on a 128^3 dam break after 240 substeps, where
    // cells hold up to 447 particles, and takes 398 so; 378 against 359 after 120; regular fluid the same.)
    for (uint32_t e = blockIdx.x; e < n;) {
        uint32_t next = 0;
        if (threadIdx.x == 0) next = gridDim.x + atomicAdd(v.p2g_list + 1, 1u);
        p2g_body<SOLVER>(v, (int)v.p2g_list[2 + e], sh);
        if (threadIdx.x == 0) part = next;
        __syncthreads();  // the next part clears the box
        e = part;
        __syncthreads();
    }
}

// u = num / weight where weight > 0 (pic_simulator.cpp:414-436); FLIP also snapshots the result.
template <bool FLIP>
__device__ __forceinline__ float4 normalize4(float4 n, float4 d)
{
    return make_float4(d.x > 0.f ? n.x / d.x : n.x, d.y > 0.f ? n.y / d.y : n.y, d.z > 0.f ? n.z / d.z : n.z,
                       d.w > 0.f ? n.w / d.w : n.w);
}

// The three components are contiguous in every face buffer (u | v | w), so the pass runs over one flat range of
// `total` faces, four per thread with 16-byte accesses when the buffers are 16-byte aligned (they start on the
// allocator's 256-byte boundaries), else face by face.
template <bool FLIP>
__device__ __forceinline__ void normalize_body(const SceneView& v, size_t total, uint32_t blk)
{
    const size_t q = blk * (size_t)blockDim.x + threadIdx.x;
    const size_t f0 = 4 * q;
    if (f0 >= total) return;
    const bool vec = ((reinterpret_cast<uintptr_t>(v.nu) | reinterpret_cast<uintptr_t>(v.du) |
                       reinterpret_cast<uintptr_t>(v.u) | reinterpret_cast<uintptr_t>(v.su)) & 15u) == 0;
    if (vec && f0 + 4 <= total) {
        const float4 o = normalize4<FLIP>(reinterpret_cast<const float4*>(v.nu)[q],
                                          reinterpret_cast<const float4*>(v.du)[q]);
        reinterpret_cast<float4*>(v.u)[q] = o;
        if (FLIP) reinterpret_cast<float4*>(v.su)[q] = o;
        return;
    }
    for (size_t f = f0; f < f0 + 4 && f < total; ++f) {
        const float d = v.du[f];
        const float val = d > 0.f ? v.nu[f] / d : v.nu[f];
        v.u[f] = val;
        if (FLIP) v.su[f] = val;
    }
}
template <bool FLIP>
__global__ void __launch_bounds__(256) k_p2g_normalize(SceneView v, size_t total)
{
    normalize_body<FLIP>(v, total, blockIdx.x);
}

// ---- flat multi-scene forms (BatchPlan, fe_internal.cuh): every scene's tiles in one launch, each block running
// its scene's transfer kind
__global__ void __launch_bounds__(kP2gThreads, 2) k_multi_p2g(const BatchPlan* __restrict__ plan)
{
    __shared__ P2gShared sh;
    __shared__ SceneView v;
    uint32_t b;
    const int s = batch_scene_of(plan, kBkP2g, b);
    stage_view(v, plan->sc[s].dst);
    if (v.solver == FE_SOLVER_PIC) p2g_body<FE_SOLVER_PIC>(v, (int)b, sh);
    else if (v.solver == FE_SOLVER_FLIP) p2g_body<FE_SOLVER_FLIP>(v, (int)b, sh);
    else p2g_body<FE_SOLVER_APIC>(v, (int)b, sh);
}

__global__ void __launch_bounds__(256) k_multi_p2g_normalize(const BatchPlan* __restrict__ plan)
{
    uint32_t b;
    const int s = batch_scene_of(plan, kBkNormalize, b);
    const SceneView& v = plan->sc[s].dst;
    const size_t total = (size_t)(v.g.nx + 1) * v.g.ny * v.g.nz + (size_t)v.g.nx * (v.g.ny + 1) * v.g.nz +
                         (size_t)v.g.nx * v.g.ny * (v.g.nz + 1);
    if (v.solver == FE_SOLVER_FLIP) normalize_body<true>(v, total, b);
    else normalize_body<false>(v, total, b);
}

}  // namespace

// Every scene's splat (accumulators cleared by launch_multi_clear) and normalisation: launch_p2g's passes.
cudaError_t launch_multi_p2g(const BatchLaunch& L, cudaStream_t st)
{
    if (L.total[kBkP2g]) {
        k_multi_p2g<<<L.total[kBkP2g], kP2gThreads, 0, st>>>(L.plan);
        count_launch();
    }
    k_multi_p2g_normalize<<<L.total[kBkNormalize], 256, 0, st>>>(L.plan);
    count_launch();
    return cudaGetLastError();
}

uint32_t p2g_blocks(const SceneView& v) { return (uint32_t)(v.g.tnx * v.g.tny * v.g.tnz) * kP2gParts; }

cudaError_t launch_p2g(const SceneView& v, cudaStream_t st)
{
    const size_t nu = (size_t)(v.g.nx + 1) * v.g.ny * v.g.nz, nvv = (size_t)v.g.nx * (v.g.ny + 1) * v.g.nz,
                 nww = (size_t)v.g.nx * v.g.ny * (v.g.nz + 1);
    cudaError_t e;
    // accumulators: numerator and weight arrays are laid out back to back, markers too (fe_scene.cu)
    if ((e = cudaMemsetAsync(v.nu, 0, (nu + nvv + nww) * sizeof(float), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(v.du, 0, (nu + nvv + nww) * sizeof(float), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(v.mu, 0, nu + nvv + nww, st)) != cudaSuccess) return e;
    if (v.np > 0) {
        const int parts = (int)p2g_blocks(v);
        if ((e = cudaMemsetAsync(v.p2g_list, 0, 2 * sizeof(uint32_t), st)) != cudaSuccess) return e;
        const unsigned few = (unsigned)((parts + 7) / 8);
        // persistent blocks: as many as are resident at once (3 per SM, APIC 2)
        const unsigned grid = (unsigned)std::min(parts, 148 * (v.solver == FE_SOLVER_APIC ? 2 : 3));
        if (v.solver == FE_SOLVER_PIC) {
            k_p2g_few<FE_SOLVER_PIC><<<few, 256, 0, st>>>(v, parts);
            k_p2g<FE_SOLVER_PIC><<<grid, kP2gThreads, 0, st>>>(v);
        } else if (v.solver == FE_SOLVER_FLIP) {
            k_p2g_few<FE_SOLVER_FLIP><<<few, 256, 0, st>>>(v, parts);
            k_p2g<FE_SOLVER_FLIP><<<grid, kP2gThreads, 0, st>>>(v);
        } else {
            k_p2g_few<FE_SOLVER_APIC><<<few, 256, 0, st>>>(v, parts);
            k_p2g<FE_SOLVER_APIC><<<grid, kP2gThreads, 0, st>>>(v);
        }
        count_launch(2);
    }
    const size_t total = nu + nvv + nww;
    const unsigned nb = (unsigned)((total + 1023) / 1024);
    if (v.solver == FE_SOLVER_FLIP) k_p2g_normalize<true><<<nb, 256, 0, st>>>(v, total);
    else k_p2g_normalize<false><<<nb, 256, 0, st>>>(v, total);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fe
