// fe_g2p.cu -- grid -> particle transfer fused with advection (K_g2p_adv).
//
// Reference: TransferGrid2Particles of PICSimulator (pic_simulator.cpp:439-450: v = Sample(grid, x)),
// FLIPSimulator (flip_simulator.cpp:121-161: v = Lerp(v + Sample(grid - snapshot, x), Sample(grid, x),
// blend)) and APICSimulator (apic_simulator.cpp:120-176: v = Sample(grid, x), C rows = sum of gradient
// weights (common/math_utils.hpp:114-176) times face values at the position clamped by h/2 on the
// transverse axes, with the CELL count as clamp size); then PICSimulator::MoveParticles
// (pic_simulator.cpp:239-312): max(maxCfl, 1) RK2 midpoint sub-steps on the GRID velocity, clamp to the
// domain box with the clamped component of the particle velocity set to 0.
//
// One thread per particle over the sorted arrays: the particle state is read once and written once
// (FP32), the grid gathers hit L1/L2 because neighbouring threads hold neighbouring particles.
#include "fe_internal.cuh"

namespace fe {
namespace {

// Stencil of a point on one staggered grid: the first face of each axis' pair and the fractions.  A pair is always two
// neighbouring faces: GetBarycentric's clamps keep the first one below the last face, and no axis has fewer than two.
struct Corner {
    int i, j, k;
    float fx, fy, fz;
};

// Two FP32 values in a register pair: the packed multiply and FMA take one instruction for both.
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(F2 s, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(s)); }
// (1 - f) a + f b of both, m = (1 - f, 1 - f) and f2 = (f, f)
__device__ __forceinline__ F2 lerp2(F2 a, F2 b, F2 m, F2 f2)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(m), "l"(a));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2), "l"(b), "l"(r));
    return r;
}

// Face values of the six arrays a transfer reads (u, v, w and the FLIP snapshot su, sv, sw).
struct FaceSource {
    const float* g[6];          // u, v, w, su, sv, sw
    int sx[3], sy[3];           // face-array sizes of the components (x, y)
    __device__ __forceinline__ size_t corner_base(int comp, const Corner& st) const
    {
        return idx3(st.i, st.j, st.k, sx[comp], sy[comp]);
    }
    // the 8 corner values of array a from its base, in the reference's corner order (x fastest): four rows of two
    __device__ __forceinline__ void load8(int a, size_t base, float c[8]) const
    {
        const float* p = g[a] + base;
        const float* q = p + sx[a % 3];
        const float* r = p + (size_t)sx[a % 3] * (size_t)sy[a % 3];
        const float* t = q + (size_t)sx[a % 3] * (size_t)sy[a % 3];
        c[0] = __ldg(p);
        c[1] = __ldg(p + 1);
        c[2] = __ldg(q);
        c[3] = __ldg(q + 1);
        c[4] = __ldg(r);
        c[5] = __ldg(r + 1);
        c[6] = __ldg(t);
        c[7] = __ldg(t + 1);
    }
    __device__ __forceinline__ void corners(int comp, const Corner& st, float c[8]) const
    {
        load8(comp, corner_base(comp, st), c);
    }
    // the corner values and their differences from the snapshot's, side by side
    __device__ __forceinline__ void corners_diff(int comp, const Corner& st, F2 c[8]) const
    {
        float a[8], b[8];
        const size_t base = corner_base(comp, st);  // the grid and its snapshot share the layout
        load8(comp, base, a);
        load8(comp + 3, base, b);
#pragma unroll
        for (int t = 0; t < 8; ++t) c[t] = pack2(a[t], a[t] - b[t]);
    }
};

// Trilinear value of the corners, the two z planes side by side.
__device__ __forceinline__ float lerp8(const float c[8], const Corner& s)
{
    const F2 mx = pack2(1.f - s.fx, 1.f - s.fx), fx = pack2(s.fx, s.fx), my = pack2(1.f - s.fy, 1.f - s.fy), fy = pack2(s.fy, s.fy);
    const F2 y0 = lerp2(pack2(c[0], c[4]), pack2(c[1], c[5]), mx, fx), y1 = lerp2(pack2(c[2], c[6]), pack2(c[3], c[7]), mx, fx);
    float b0, b1;
    unpack2(lerp2(y0, y1, my, fy), b0, b1);
    return lerpf_ref(b0, b1, s.fz);
}
// ... of both values of each corner.
__device__ __forceinline__ void lerp8x2(const F2 c[8], const Corner& s, float& first, float& second)
{
    const F2 mx = pack2(1.f - s.fx, 1.f - s.fx), fx = pack2(s.fx, s.fx), my = pack2(1.f - s.fy, 1.f - s.fy), fy = pack2(s.fy, s.fy);
    F2 z[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
        z[k] = lerp2(lerp2(c[4 * k], c[4 * k + 1], mx, fx), lerp2(c[4 * k + 2], c[4 * k + 3], mx, fx), my, fy);
    unpack2(lerp2(z[0], z[1], pack2(1.f - s.fz, 1.f - s.fz), pack2(s.fz, s.fz)), first, second);
}

// GetBarycentric index and fraction of a point along one axis of one staggered grid, bary()'s cases by clamping: the
// position between the first and the last face (NaN: the first), its floor below the last.
struct AxisFrac {
    int i;
    float f;
};
__device__ __forceinline__ AxisFrac axis_frac(float x, float o, float ih, int size)
{
    const float t = fminf(fmaxf((x - o) * ih, 0.f), (float)(size - 1));
    const float s = fminf(floorf(t), (float)(size - 2));
    AxisFrac a;
    a.i = (int)s;
    a.f = t - s;
    return a;
}
__device__ __forceinline__ Corner stencil_of(const AxisFrac& a, const AxisFrac& b, const AxisFrac& c)
{
    Corner s;
    s.i = a.i; s.fx = a.f;
    s.j = b.i; s.fy = b.f;
    s.k = c.i; s.fz = c.f;
    return s;
}

// The three staggered grids' stencils at one point, as stencil() gives them.  Along each axis the two grids that are
// not staggered along it have the same data origin (both offset by half a cell, set side by side with the scene:
// xo[1] == zo[1], yo[0] == zo[0], xo[2] == yo[2], and likewise for the FLIP residual origins) and the same size, so
// their index and fraction are one computation: 6 per point instead of 9.
__device__ __forceinline__ void stencils3(float x, float y, float z, const float ou[3], const float ov[3],
                                          const float ow[3], const float ih[3], int nx, int ny, int nz, Corner& su,
                                          Corner& sv, Corner& sw)
{
    const AxisFrac xf = axis_frac(x, ou[0], ih[0], nx + 1), xc = axis_frac(x, ov[0], ih[0], nx);
    const AxisFrac yf = axis_frac(y, ov[1], ih[1], ny + 1), yc = axis_frac(y, ou[1], ih[1], ny);
    const AxisFrac zf = axis_frac(z, ow[2], ih[2], nz + 1), zc = axis_frac(z, ou[2], ih[2], nz);
    su = stencil_of(xf, yc, zc);
    sv = stencil_of(xc, yf, zc);
    sw = stencil_of(xc, yc, zf);
}

// The grid velocity at a point: the three components' trilinear samples, each stencil built just before its loads
// (the shared fractions of stencils3 carried from one component to the next).
__device__ __forceinline__ void sample_vel(const SceneView& v, const FaceSource& fs, float x, float y, float z,
                                           float out[3])
{
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const float* ih = v.inv_hf;
    float c[8];
    const AxisFrac xf = axis_frac(x, v.xo[0], ih[0], nx + 1);
    const AxisFrac yc = axis_frac(y, v.xo[1], ih[1], ny);
    const AxisFrac zc = axis_frac(z, v.xo[2], ih[2], nz);
    const Corner su = stencil_of(xf, yc, zc);
    fs.corners(0, su, c);
    out[0] = lerp8(c, su);
    const AxisFrac xc = axis_frac(x, v.yo[0], ih[0], nx);
    const AxisFrac yf = axis_frac(y, v.yo[1], ih[1], ny + 1);
    const Corner sv = stencil_of(xc, yf, zc);
    fs.corners(1, sv, c);
    out[1] = lerp8(c, sv);
    const AxisFrac zf = axis_frac(z, v.zo[2], ih[2], nz + 1);
    const Corner sw = stencil_of(xc, yc, zf);
    fs.corners(2, sw, c);
    out[2] = lerp8(c, sw);
}

// Trilinear sample of (grid - snapshot) with the reference's Lerp tree (the FLIP residual grid,
// flip_simulator.cpp:138-150), and of the grid itself at the same stencil from the same face values.
__device__ __forceinline__ float sample_diff(const FaceSource& fs, int comp, const Corner& s, float& plain)
{
    F2 c[8];
    fs.corners_diff(comp, s, c);
    float diff;
    lerp8x2(c, s, plain, diff);
    return diff;
}

// sum_t gradweight_t * face_t for one velocity component (apic_simulator.cpp:311-336) from the stencil's 8 corner values:
// per axis the differences of the corners along it, interpolated along the others, over h.  Returns the trilinear value,
// whose partial sums the rows share.
__device__ __forceinline__ float apic_row_vals(const float c[8], const Corner& s, const float ih[3], float out[3])
{
    const F2 mx = pack2(1.f - s.fx, 1.f - s.fx), fx = pack2(s.fx, s.fx), my = pack2(1.f - s.fy, 1.f - s.fy), fy = pack2(s.fy, s.fy);
    const F2 y0 = lerp2(pack2(c[0], c[4]), pack2(c[1], c[5]), mx, fx), y1 = lerp2(pack2(c[2], c[6]), pack2(c[3], c[7]), mx, fx);
    float x0, x1;  // along x, lower and upper z plane
    unpack2(lerp2(pack2(c[1] - c[0], c[5] - c[4]), pack2(c[3] - c[2], c[7] - c[6]), my, fy), x0, x1);
    float a0, a1, e0, e1, b0, b1;
    unpack2(y0, a0, a1);
    unpack2(y1, e0, e1);
    unpack2(lerp2(y0, y1, my, fy), b0, b1);
    out[0] = ih[0] * lerpf_ref(x0, x1, s.fz);
    out[1] = ih[1] * lerpf_ref(e0 - a0, e1 - a1, s.fz);
    out[2] = ih[2] * (b1 - b0);
    return lerpf_ref(b0, b1, s.fz);
}

// APIC: component c's grid sample at the particle (stencil s, the velocity grid's face counts as sizes) and its C row.
// The row's stencil is taken at the particle clamped by h/2 on the two transverse axes with the CELL counts as sizes;
// where no clamp moves the particle and its index along the component's own axis is below n - 1 (the two sizes then
// give the same GetBarycentric result), it is s itself, and the row reuses the sample's 8 corner values.
__device__ __forceinline__ float apic_component(const SceneView& v, const FaceSource& fs, int c, const Corner& s,
                                                const float P[3], const float lo[3], const float hi[3], uint64_t p)
{
    float c8[8];
    fs.corners(c, s, c8);
    float row[3];
    const float pic = apic_row_vals(c8, s, v.inv_hf, row);
    float q[3] = {P[0], P[1], P[2]};
#pragma unroll
    for (int a = 0; a < 3; ++a)
        if (a != c) q[a] = q[a] < lo[a] ? lo[a] : (q[a] > hi[a] ? hi[a] : q[a]);
    const int n_c = c == 0 ? v.g.nx : (c == 1 ? v.g.ny : v.g.nz);
    const int i_c = c == 0 ? s.i : (c == 1 ? s.j : s.k);
    if (!(q[0] == P[0] && q[1] == P[1] && q[2] == P[2] && i_c <= n_c - 2)) {
        const float* org = c == 0 ? v.xo : (c == 1 ? v.yo : v.zo);
        const Corner t = stencil_of(axis_frac(q[0], org[0], v.inv_hf[0], v.g.nx), axis_frac(q[1], org[1], v.inv_hf[1], v.g.ny),
                                    axis_frac(q[2], org[2], v.inv_hf[2], v.g.nz));
        fs.corners(c, t, c8);
        apic_row_vals(c8, t, v.inv_hf, row);
    }
    v.c[3 * c][p] = row[0];
    v.c[3 * c + 1][p] = row[1];
    v.c[3 * c + 2][p] = row[2];
    return pic;
}

// APIC's transfer at the particle: the grid velocity (as sample_vel) and the three C rows.
__device__ __forceinline__ void sample_vel_apic(const SceneView& v, const FaceSource& fs, float x, float y, float z,
                                                uint64_t p, float out[3])
{
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const float* ih = v.inv_hf;
    const float lo[3] = {v.originf[0] + 0.5f * v.hf[0], v.originf[1] + 0.5f * v.hf[1], v.originf[2] + 0.5f * v.hf[2]};
    const float hi[3] = {v.originf[0] + v.sizef[0] - 0.5f * v.hf[0], v.originf[1] + v.sizef[1] - 0.5f * v.hf[1],
                         v.originf[2] + v.sizef[2] - 0.5f * v.hf[2]};
    const float P[3] = {x, y, z};
    const AxisFrac xf = axis_frac(x, v.xo[0], ih[0], nx + 1);
    const AxisFrac yc = axis_frac(y, v.xo[1], ih[1], ny);
    const AxisFrac zc = axis_frac(z, v.xo[2], ih[2], nz);
    out[0] = apic_component(v, fs, 0, stencil_of(xf, yc, zc), P, lo, hi, p);
    const AxisFrac xc = axis_frac(x, v.yo[0], ih[0], nx);
    const AxisFrac yf = axis_frac(y, v.yo[1], ih[1], ny + 1);
    out[1] = apic_component(v, fs, 1, stencil_of(xc, yf, zc), P, lo, hi, p);
    const AxisFrac zf = axis_frac(z, v.zo[2], ih[2], nz + 1);
    out[2] = apic_component(v, fs, 2, stencil_of(xc, yc, zf), P, lo, hi, p);
}

// The transfer and move of particle p (pic_simulator.cpp:239-312, flip_simulator.cpp:121-161,
// apic_simulator.cpp:120-176), reading face values through fs.
template <int SOLVER, bool G2P, bool MOVE>
__device__ __forceinline__ void g2p_particle(const SceneView& v, const G2PArgs& g, const FaceSource& fs, uint64_t p)
{
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const float x = v.px[p], y = v.py[p], z = v.pz[p];
    float vel[3];
    float pic[3];
    bool have_pic = false;
    if (G2P) {
        if (SOLVER == FE_SOLVER_FLIP) {
            Corner su, sv, sw;
            stencils3(x, y, z, v.rxo, v.ryo, v.rzo, v.inv_hf, nx, ny, nz, su, sv, sw);
            const bool share = g.same_origins && v.blend > 0.f;
            float flip[3] = {v.vx[p] + sample_diff(fs, 0, su, pic[0]), v.vy[p] + sample_diff(fs, 1, sv, pic[1]),
                             v.vz[p] + sample_diff(fs, 2, sw, pic[2])};
            if (v.blend > 0.f) {
                if (!share) sample_vel(v, fs, x, y, z, pic);
                have_pic = true;
#pragma unroll
                for (int a = 0; a < 3; ++a) flip[a] = (1.f - v.blend) * flip[a] + v.blend * pic[a];
            }
            vel[0] = flip[0];
            vel[1] = flip[1];
            vel[2] = flip[2];
        } else {
            if (SOLVER == FE_SOLVER_APIC) sample_vel_apic(v, fs, x, y, z, p, pic);
            else sample_vel(v, fs, x, y, z, pic);
            have_pic = true;
            vel[0] = pic[0];
            vel[1] = pic[1];
            vel[2] = pic[2];
        }
    } else {
        vel[0] = v.vx[p];
        vel[1] = v.vy[p];
        vel[2] = v.vz[p];
    }
    if (MOVE) {
        float pt0[3] = {x, y, z}, pt1[3] = {x, y, z};
        const float half = 0.5f * g.dt_sub;
        for (int t = 0; t < g.nsub; ++t) {
            float v0[3], vm[3];
            if (t == 0 && have_pic) {
                v0[0] = pic[0]; v0[1] = pic[1]; v0[2] = pic[2];
            } else {
                sample_vel(v, fs, pt0[0], pt0[1], pt0[2], v0);
            }
            const float mid[3] = {pt0[0] + half * v0[0], pt0[1] + half * v0[1], pt0[2] + half * v0[2]};
            sample_vel(v, fs, mid[0], mid[1], mid[2], vm);
#pragma unroll
            for (int a = 0; a < 3; ++a) pt1[a] = pt0[a] + g.dt_sub * vm[a];
#pragma unroll
            for (int a = 0; a < 3; ++a) pt0[a] = pt1[a];
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (pt1[a] <= g.dom_lo[a]) { pt1[a] = g.dom_lo[a]; vel[a] = 0.f; }
            if (pt1[a] >= g.dom_hi[a]) { pt1[a] = g.dom_hi[a]; vel[a] = 0.f; }
            // a NaN position (diverged input) is pinned to the lower wall so keys stay in range
            if (!(pt1[a] == pt1[a])) { pt1[a] = g.dom_lo[a]; vel[a] = 0.f; }
        }
        v.px[p] = pt1[0];
        v.py[p] = pt1[1];
        v.pz[p] = pt1[2];
    }
    v.vx[p] = vel[0];
    v.vy[p] = vel[1];
    v.vz[p] = vel[2];
}

__device__ __forceinline__ FaceSource global_source(const SceneView& v, const G2PArgs& g)
{
    FaceSource fs;
    fs.g[0] = g.u; fs.g[1] = g.v; fs.g[2] = g.w;
    fs.g[3] = v.su; fs.g[4] = v.sv; fs.g[5] = v.sw;
    fs.sx[0] = v.g.nx + 1; fs.sx[1] = v.g.nx; fs.sx[2] = v.g.nx;
    fs.sy[0] = v.g.ny; fs.sy[1] = v.g.ny + 1; fs.sy[2] = v.g.ny;
    return fs;
}

// One thread per particle over the sorted arrays: neighbouring threads hold neighbouring particles, so the face
// gathers hit L1/L2.  Bound by the L1's address lookups (86 % at 128^3 FLIP) and issue: 149 us there and 1596 us at 256^3
// APIC (32 M particles) with the indexes of clamped pairs, an address per corner and one sample at a time, 135 and 1225 with
// rows of two faces and packed interpolation (968 against 648 instructions a particle).  The faces of half a tile in shared
// memory (12 x 12 x 8 per component, read by the half tile's particles) took 136 and 1080, but 12 us more at 32^3.
template <int SOLVER, bool G2P, bool MOVE>
__global__ void __launch_bounds__(256, 4) k_g2p(SceneView v, G2PArgs g)
{
    const uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= v.np) return;
    g2p_particle<SOLVER, G2P, MOVE>(v, g, global_source(v, g), p);
}

// Flat multi-scene form (BatchPlan, fe_internal.cuh): every scene's particles in one launch, transfer and move
// fused, each block running its scene's transfer kind.
__global__ void __launch_bounds__(256, 4) k_multi_g2p(const BatchPlan* __restrict__ plan)
{
    __shared__ SceneView v;
    uint32_t b;
    const int s = batch_scene_of(plan, kBkPart, b);
    const BatchScene& e = plan->sc[s];
    stage_view(v, e.dst);
    const uint64_t p = b * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= v.np) return;
    if (v.solver == FE_SOLVER_PIC) g2p_particle<FE_SOLVER_PIC, true, true>(v, e.g2p, global_source(v, e.g2p), p);
    else if (v.solver == FE_SOLVER_FLIP) g2p_particle<FE_SOLVER_FLIP, true, true>(v, e.g2p, global_source(v, e.g2p), p);
    else g2p_particle<FE_SOLVER_APIC, true, true>(v, e.g2p, global_source(v, e.g2p), p);
}

template <int SOLVER>
void launch_solver(const SceneView& v, const G2PArgs& g, bool do_g2p, bool do_move, cudaStream_t st)
{
    const unsigned nb = (unsigned)((v.np + 255) / 256);
    if (do_g2p && do_move) k_g2p<SOLVER, true, true><<<nb, 256, 0, st>>>(v, g);
    else if (do_g2p) k_g2p<SOLVER, true, false><<<nb, 256, 0, st>>>(v, g);
    else k_g2p<SOLVER, false, true><<<nb, 256, 0, st>>>(v, g);
}

}  // namespace

cudaError_t launch_multi_g2p(const BatchLaunch& L, cudaStream_t st)
{
    if (!L.total[kBkPart]) return cudaSuccess;
    k_multi_g2p<<<L.total[kBkPart], 256, 0, st>>>(L.plan);
    count_launch();
    return cudaGetLastError();
}

G2PArgs g2p_args(const SceneView& v, double dt)
{
    G2PArgs g;
    g.nsub = v.rk_substeps;
    g.dt_sub = (float)(dt / g.nsub);
    g.same_origins = 1;
    for (int a = 0; a < 3; ++a)
        g.same_origins &= (v.rxo[a] == v.xo[a] && v.ryo[a] == v.yo[a] && v.rzo[a] == v.zo[a]) ? 1 : 0;
    for (int a = 0; a < 3; ++a) {
        g.dom_lo[a] = (float)v.origin[a];
        g.dom_hi[a] = (float)(v.origin[a] + v.size[a]);
    }
    g.u = v.u;  // after the post group the velocity is back in buffer A
    g.v = v.v;
    g.w = v.w;
    return g;
}

cudaError_t launch_g2p(const SceneView& v, double dt, bool do_g2p, bool do_move, cudaStream_t st)
{
    if (v.np == 0 || (!do_g2p && !do_move)) return cudaSuccess;
    const G2PArgs g = g2p_args(v, dt);
    if (v.solver == FE_SOLVER_PIC) launch_solver<FE_SOLVER_PIC>(v, g, do_g2p, do_move, st);
    else if (v.solver == FE_SOLVER_FLIP) launch_solver<FE_SOLVER_FLIP>(v, g, do_g2p, do_move, st);
    else launch_solver<FE_SOLVER_APIC>(v, g, do_g2p, do_move, st);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fe
