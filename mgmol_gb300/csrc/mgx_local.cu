// Localized orbitals: box-local storage and one persistent fused kernel for
// the fine-level work of an orbital iteration on uneven mask boxes.
//
// Orbital j lives on the level-0 box of its localization mask (origin o_j,
// extents e_j, the box form of mgx_masks: point b of the box is grid point
// (o_j + b) mod n, z fastest), packed one box after another.  Outside its
// box an orbital is zero, which is what the masks make of it on the whole
// grid: the mask values are zero there (src/GridMask.cc:120-264).
//
// The fused step, per orbital (FP32, the reference's operators):
//   r  = Mc (B(phi - V psi) + Delta_M psi)       = Mc (B phi - H psi)
//   u0 = gamma r
//   u1 = M(u0 - jf (A u0 - r))                    first Jacobi sweep
//   u2 = M(u1 - jf (A u1 - r)),  w = M(A u1 - r)  second sweep
// with H psi = -Delta_M psi + B(V psi) (Hamiltonian::applyLocal,
// src/Hamiltonian.cc:106-132), phi the column of Psi Theta (the residual of
// MGmol::computeResidualUsingHPhi, src/MGmol.cc:1227-1290, with the
// correction mask Mc of LocGridOrbitals::applyCorrMask), A = -Delta_M and
// the orbital mask M (GridMaskMax) of the V-cycle's fine-level pre-sweeps
// (Preconditioning<T>::mg, src/Preconditioning.cc:170-178).  u2 and w are
// what the V-cycle restricts next.
//
// One CTA takes (orbital, column) items from a work list until it is empty
// (largest orbitals first); a column is a window of the orbital's y and z
// marched along x, so the orbital block is read once (plus the y / z halo)
// and u2, w written once.  The threads per CTA and the CTAs per SM are chosen
// by timing (mgx_local_tune); the launch can be a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <vector>

#include "mgx_internal.cuh"
#include "mgx_stencil.cuh"

namespace mgx
{
namespace loc
{
constexpr int HALO = 3;

/* -Delta_M-like stencil: centre, faces, edges */
struct Stencil19
{
    float c0, cx, cy, cz, cxy, cyz, cxz;
};

struct StepParams
{
    const float* psi;
    const float* phi;
    const float* V; // FP32 potential on the whole grid
    float* u;
    float* w;
    const int* box;       // 6 per orbital: origin, extents
    const int* core;      // 6 per orbital: the box points with a mask that is not zero lie in
                          // [core0, core3) x [core1, core4) x [core2, core5)
    const int* range;     // per box column (y, z): they lie in x of [r & 0xffff, r >> 16); NULL:
                          // the whole box
    const size_t* roff;   // offset of an orbital's columns
    const size_t* off;    // packed offset of each orbital
    const float* mvals;   // orbital mask values, box-local
    const size_t* moff;
    const float* cvals;   // correction mask values, box-local
    const size_t* coff;
    const int4* items;    // (orbital, ty | tz << 16, column origin y, z), or (orbital, 0, 0, 0):
                          // the points outside the core
    int nitems;
    int* counter;
    int n[3];
    Stencil19 lap;        // Delta_M (stage 1)
    Stencil19 sweep;      // gamma r - jf (A gamma r - r) of r (stage 2)
    Stencil19 A;          // -Delta_M (stage 3)
    float jf;
};

__device__ __forceinline__ int wrapi(int i, int n)
{
    i %= n;
    return i < 0 ? i + n : i;
}

__device__ __forceinline__ float clampm(float v, float m)
{
    if (v > m) return m;
    if (v < -m) return -m;
    return v;
}

__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }

/* the sums of a plane at a z pair (index i, odd, of the pair's first value):
 * the pair itself, its y neighbours, its z neighbours, its y-z diagonals.
 * Six 8-byte loads: the pair lies across two of them, so that (z - 1, z) and
 * (z + 1, z + 2) add up to the z neighbours of both points at once */
struct Sums
{
    float2 a, ey, ez, q;
};
__device__ __forceinline__ Sums plane_sums(const float* A, int i, int pitch)
{
    const float2 lo = *reinterpret_cast<const float2*>(A + i - 1);
    const float2 hi = *reinterpret_cast<const float2*>(A + i + 1);
    const float2 ls = __fadd2_rn(*reinterpret_cast<const float2*>(A + i - pitch - 1),
        *reinterpret_cast<const float2*>(A + i + pitch - 1));
    const float2 hs = __fadd2_rn(*reinterpret_cast<const float2*>(A + i - pitch + 1),
        *reinterpret_cast<const float2*>(A + i + pitch + 1));
    return { make_float2(lo.y, hi.x), make_float2(ls.y, hs.x), __fadd2_rn(lo, hi),
        __fadd2_rn(ls, hs) };
}

/* what a plane adds to the stencil of the planes beside it (side) and, with g the
 * share of the plane before, to its own (mid: the centre, the largest term, last) */
__device__ __forceinline__ float2 side(const Sums& t, const Stencil19& c)
{
    return __ffma2_rn(f2(c.cxz), t.ez, __ffma2_rn(f2(c.cxy), t.ey, __fmul2_rn(f2(c.cx), t.a)));
}
__device__ __forceinline__ float2 mid(const Sums& t, const Stencil19& c, float2 g)
{
    return __ffma2_rn(f2(c.c0), t.a,
        __ffma2_rn(f2(c.cy), t.ey, __ffma2_rn(f2(c.cz), t.ez, __ffma2_rn(f2(c.cyz), t.q, g))));
}

/* one periodic coordinate of a box point: b in [-3, e + 3) with e + 6 <= n */
__device__ __forceinline__ int wrap1(int g, int n)
{
    return g < 0 ? g + n : (g >= n ? g - n : g);
}

/* A CTA owns a ty x tz column of an orbital's core -- the part of its box
 * where a mask is not zero, outside of which u = w = 0 -- and marches along x.
 * Thread (y, z pair) of the column and its halo of 3 keeps its place in all
 * four stages.  At step s, with p = xa - 3 + s:
 *   stage 0 stores psi and d = phi - V psi of plane p,
 *   stage 1 reads plane p - 1 of both and completes r of plane p - 2,
 *   stage 2 reads plane p - 3 of r and completes u1 of plane p - 4,
 *   stage 3 reads plane p - 5 of u1 and completes u, w of plane p - 6:
 * every stage reads what was stored before the last barrier, so there is one
 * barrier per step and two planes per array.  The stencil along x is
 * accumulated: a plane's sums are formed once and give a share to three
 * planes (Sums, side, mid).  The results next to the edge of the halo are
 * made from values that were never set; no stage's valid region, one point
 * narrower than that of the stage before, reads them.
 *
 * The inputs of the next step are loaded one step ahead.  A thread skips the
 * planes that no mask value of its pair reaches (P.range), and does not load
 * there.  Two steps per turn of the loop: the queues of r, u1 and the masks
 * then need no moves.
 *
 * Why this form: 1536 orbitals on 160^3 (radii 4 to 8 bohr at h = 0.3; 4.4 GB,
 * 0.65 ms at the copy rate) took 3.90 ms with a kernel that marched the whole
 * box, mapped each stage's region to the threads anew (three barriers per
 * plane, up to half of the threads idle in a stage's last pass, 36
 * shared-memory wavefronts per stencil, mask values loaded where they were
 * used: 15 % of the issue slots, long scoreboard first).  Only the core of the
 * boxes: 3.39 ms.  This kernel: 1.96 ms with 448 threads and 2 CTAs per SM (2.36
 * with one step per turn), 59 % of the issue slots, DRAM at 28 %: bound by
 * instruction issue and, at 24 of 32 lanes, by the halo. */
template <int NT> struct Plane
{
    // the column with its halo: at most 2 NT values, and two more per row
    // (rows of eight values or more: at most NT / 4 of them)
    static constexpr int SIZE = 2 * NT + NT / 2;
    static constexpr size_t SMEM = 8 * SIZE * sizeof(float);
};

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) local_step_kernel(const StepParams P)
{
    constexpr int PLANE = Plane<NT>::SIZE;
    extern __shared__ __align__(16) float sm[]; // two planes each of psi, d, r, u1
    __shared__ int s_item;
    const int tid = threadIdx.x;
    for (;;)
    {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(P.counter, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= P.nitems) break;
        const int4 W = P.items[it]; // (orbital, ty | tz << 16, y0, z0)
        const int f  = W.x;
        const int ty = W.y & 0xffff, tz = W.y >> 16, y0 = W.z, z0 = W.w;
        const int* b = P.box + 6 * f;
        const int o0 = b[0], o1 = b[1], o2 = b[2], e0 = b[3], e1 = b[4], e2 = b[5];
        const int* core = P.core + 6 * f;
        const int xa = core[0], xb = core[3], yb = core[4], zb = core[5];
        float* const ub = P.u + P.off[f];
        float* const wb = P.w + P.off[f];
        if (ty == 0)
        {
            // u = w = 0 outside the core, a warp per z row
            const int ya = core[1], za = core[2];
            for (int r = tid / 32; r < e0 * e1; r += NT / 32)
            {
                const int x = r / e1, y = r - x * e1;
                const bool cut = x >= xa && x < xb && y >= ya && y < yb;
                const size_t o = (size_t)r * e2;
                for (int z = tid & 31; z < e2; z += 32)
                    if (!(cut && z >= za && z < zb))
                    {
                        ub[o + z] = 0.f;
                        wb[o + z] = 0.f;
                    }
            }
            continue;
        }
        const int z3 = tz + 2 * HALO, pitch = z3 + 2, rows = ty + 2 * HALO, np = z3 / 2;
        const int qy = tid / np, qz = 2 * (tid - qy * np);
        const int by = y0 + qy - HALO, bz = z0 + qz - HALO;
        const int i  = qy * pitch + qz + 1;
        const bool on  = qy < rows;
        const bool on1 = qy >= 1 && qy < rows - 1, on2 = qy >= 2 && qy < rows - 2;
        const bool on3 = qy >= 3 && qy < rows - 3;
        // the pair's points in the box, and among those that this column stores
        const bool in0 = on && by >= 0 && by < e1 && bz >= 0 && bz < e2;
        const bool in1 = on && by >= 0 && by < e1 && bz + 1 >= 0 && bz + 1 < e2;
        const bool st0 = on3 && by < yb && bz >= z0 && bz < min(z0 + tz, zb);
        const bool st1 = on3 && by < yb && bz + 1 >= z0 && bz + 1 < min(z0 + tz, zb);
        // planes [lo, hi) with a mask value at the pair, [llo, lhi) with one at a neighbour
        int lo = 1 << 20, hi = 0, llo = 1 << 20, lhi = 0;
        if (P.range)
        {
            const int* rg = P.range + P.roff[f];
            if (on)
                for (int dy = -1; dy <= 1; dy++)
                    for (int dz = -1; dz <= 2; dz++)
                    {
                        const int y = by + dy, z = bz + dz;
                        if (y < 0 || y >= e1 || z < 0 || z >= e2) continue;
                        const int r = rg[y * e2 + z], l = r & 0xffff, h = r >> 16;
                        if (l >= h) continue;
                        llo = min(llo, max(l - 1, 0));
                        lhi = max(lhi, min(h + 1, e0));
                        if (dy == 0 && (dz == 0 || dz == 1))
                        {
                            lo = min(lo, l);
                            hi = max(hi, h);
                        }
                    }
        }
        else if (in0 || in1)
        {
            lo = llo = 0;
            hi = lhi = e0;
        }
        const int ex = e1 * e2;
        const int li      = by * e2 + bz;
        const int gy      = wrap1(o1 + by, P.n[1]);
        const int v0      = gy * P.n[2] + wrap1(o2 + bz, P.n[2]);
        const int v1      = gy * P.n[2] + wrap1(o2 + bz + 1, P.n[2]);
        const float* psi  = P.psi + P.off[f];
        const float* phi  = P.phi + P.off[f];
        const float* mo   = P.mvals + P.moff[f];
        const float* mc   = P.cvals + P.coff[f];
        const size_t vx   = (size_t)P.n[1] * P.n[2];
        float2 rps, rph, rv, rmc, rmo; // of the next step
        auto load = [&](int p) {
            rps = rph = rv = rmc = rmo = f2(0.f);
            if (p >= llo && p < lhi)
            {
                const float* V = P.V + wrap1(o0 + p, P.n[0]) * vx;
                const size_t q = (size_t)p * ex;
                const float *psp = psi + q, *php = phi + q;
                if (in0)
                {
                    rps.x = psp[li];
                    rph.x = php[li];
                    rv.x  = V[v0];
                }
                if (in1)
                {
                    rps.y = psp[li + 1];
                    rph.y = php[li + 1];
                    rv.y  = V[v1];
                }
            }
            if (p - 2 >= lo && p - 2 < hi)
            {
                const float* m = mc + (size_t)(p - 2) * ex;
                if (in0) rmc.x = m[li];
                if (in1) rmc.y = m[li + 1];
            }
            if (p - 4 >= lo && p - 4 < hi)
            {
                const float* m = mo + (size_t)(p - 4) * ex;
                if (in0) rmo.x = m[li];
                if (in1) rmo.y = m[li + 1];
            }
        };
        load(xa - 3);
        float2 acc1 = f2(0.f), g1 = f2(0.f), acc2 = f2(0.f), g2 = f2(0.f), acc3 = f2(0.f),
               g3 = f2(0.f);
        float2 ra1 = f2(0.f), ra2 = f2(0.f), ua1 = f2(0.f), mo1 = f2(0.f), mo2 = f2(0.f);
        const int steps = xb - xa + 9;
#pragma unroll 2
        for (int s = 0; s < steps; s++)
        {
            const int p     = xa - 3 + s;
            float* const wr = sm + (s & 1) * PLANE;
            const float* rd = sm + (1 - (s & 1)) * PLANE;
            if (on)
            {
                const float2 mcp = rmc, mo0 = rmo;
                const float2 d = __ffma2_rn(make_float2(-rv.x, -rv.y), rps, rph);
                wr[i]             = rps.x;
                wr[i + 1]         = rps.y;
                wr[2 * PLANE + i]     = d.x;
                wr[2 * PLANE + i + 1] = d.y;
                load(p + 1);
                if (on1)
                {
                    float2 r = f2(0.f);
                    if (p - 1 >= lo - 1 && p - 1 < hi + 1)
                    {
                        const Sums t = plane_sums(rd, i, pitch);
                        const Sums v = plane_sums(rd + 2 * PLANE, i, pitch);
                        const float2 g = __ffma2_rn(f2(1.f / 12.f), v.a, side(t, P.lap));
                        const float2 m = __ffma2_rn(f2(1.f / 12.f), __fadd2_rn(v.ey, v.ez),
                            __ffma2_rn(f2(0.5f), v.a, g1));
                        const float2 o = __fadd2_rn(acc1, g);
                        acc1 = mid(t, P.lap, m);
                        g1   = g;
                        r    = make_float2(mcp.x != 0.f ? mcp.x * o.x : 0.f,
                            mcp.y != 0.f ? mcp.y * o.y : 0.f);
                    }
                    wr[4 * PLANE + i]     = r.x;
                    wr[4 * PLANE + i + 1] = r.y;
                }
                if (on2)
                {
                    float2 u = f2(0.f), ra = f2(0.f);
                    if (p - 3 >= lo - 1 && p - 3 < hi + 1)
                    {
                        const Sums t   = plane_sums(rd + 4 * PLANE, i, pitch);
                        const float2 g = side(t, P.sweep);
                        const float2 o = __fadd2_rn(acc2, g);
                        acc2 = mid(t, P.sweep, g2);
                        g2   = g;
                        ra   = t.a;
                        u = make_float2(mo0.x != 0.f ? clampm(o.x, mo0.x) : 0.f,
                            mo0.y != 0.f ? clampm(o.y, mo0.y) : 0.f);
                    }
                    wr[6 * PLANE + i]     = u.x;
                    wr[6 * PLANE + i + 1] = u.y;
                    if (on3)
                    {
                        float2 w = f2(0.f), v = f2(0.f);
                        if (p - 5 >= lo - 1 && p - 5 < hi + 1)
                        {
                            const Sums t   = plane_sums(rd + 6 * PLANE, i, pitch);
                            const float2 g = side(t, P.A);
                            const float2 o = __fadd2_rn(acc3, g);
                            // A u1 - r: the residual of plane p - 5 goes in here
                            acc3 = mid(t, P.A, __fadd2_rn(make_float2(-ra2.x, -ra2.y), g3));
                            g3   = g;
                            const float2 x = __ffma2_rn(f2(-P.jf), o, ua1);
                            if (mo2.x != 0.f) { w.x = clampm(o.x, mo2.x); v.x = clampm(x.x, mo2.x); }
                            if (mo2.y != 0.f) { w.y = clampm(o.y, mo2.y); v.y = clampm(x.y, mo2.y); }
                            ua1 = t.a;
                        }
                        if (p - 6 >= xa)
                        {
                            float* const up = ub + (size_t)(p - 6) * ex;
                            float* const wp = wb + (size_t)(p - 6) * ex;
                            if (st0)
                            {
                                up[li] = v.x;
                                wp[li] = w.x;
                            }
                            if (st1)
                            {
                                up[li + 1] = v.y;
                                wp[li + 1] = w.y;
                            }
                        }
                    }
                    ra2 = ra1;
                    ra1 = ra;
                    mo2 = mo1;
                    mo1 = mo0;
                }
            }
            __syncthreads();
        }
    }
}

/* what the masks of an orbital (blockIdx.x) reach: per box column (y, z) the
 * range [lo, hi) of x with a value of either mask that is not zero, lo | hi <<
 * 16 (none: 0), and the bounds of all of them (none: all zero) */
__global__ void __launch_bounds__(256) core_kernel(const float* __restrict__ mvals,
    const size_t* __restrict__ moff, const float* __restrict__ cvals,
    const size_t* __restrict__ coff, const int* __restrict__ box, const size_t* __restrict__ roff,
    int* __restrict__ range, int* __restrict__ core)
{
    __shared__ int lo[3], hi[3];
    const int f  = blockIdx.x;
    const int* b = box + 6 * f;
    if (threadIdx.x < 3)
    {
        lo[threadIdx.x] = 1 << 20;
        hi[threadIdx.x] = 0;
    }
    __syncthreads();
    const float* m = mvals + moff[f];
    const float* c = cvals + coff[f];
    const int ex   = b[4] * b[5];
    for (int i = threadIdx.x; i < ex; i += blockDim.x)
    {
        int l = 1 << 20, h = 0;
        for (int x = 0; x < b[3]; x++)
        {
            const size_t k = (size_t)x * ex + i;
            // (NaN counts as a value)
            if (!(m[k] == 0.f && c[k] == 0.f))
            {
                l = min(l, x);
                h = x + 1;
            }
        }
        range[roff[f] + i] = h ? (l | (h << 16)) : 0;
        if (h)
        {
            atomicMin(lo, l);
            atomicMax(hi, h);
            atomicMin(lo + 1, i / b[5]);
            atomicMax(hi + 1, i / b[5] + 1);
            atomicMin(lo + 2, i % b[5]);
            atomicMax(hi + 2, i % b[5] + 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3)
    {
        core[6 * f + threadIdx.x]     = hi[threadIdx.x] ? lo[threadIdx.x] : 0;
        core[6 * f + 3 + threadIdx.x] = hi[threadIdx.x];
    }
}

/* packed box-local <-> whole-grid copies (blockIdx.y = orbital) */
__global__ void __launch_bounds__(256) gather_kernel(const float* __restrict__ full, size_t ld,
    float* __restrict__ packed, const int* __restrict__ box, const size_t* __restrict__ off,
    int n0, int n1, int n2)
{
    const int f  = blockIdx.y;
    const int* b = box + 6 * f;
    const size_t vol = (size_t)b[3] * b[4] * b[5];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < vol;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const int bz = (int)(i % b[5]), by = (int)((i / b[5]) % b[4]), bx = (int)(i / ((size_t)b[5] * b[4]));
        const int gx = wrapi(b[0] + bx, n0), gy = wrapi(b[1] + by, n1), gz = wrapi(b[2] + bz, n2);
        packed[off[f] + i] = full[(size_t)f * ld + ((size_t)gx * n1 + gy) * n2 + gz];
    }
}

__global__ void __launch_bounds__(256) scatter_kernel(const float* __restrict__ packed,
    float* __restrict__ full, size_t ld, const int* __restrict__ box,
    const size_t* __restrict__ off, int n0, int n1, int n2)
{
    const int f  = blockIdx.y;
    const int* b = box + 6 * f;
    const size_t vol = (size_t)b[3] * b[4] * b[5];
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < vol;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const int bz = (int)(i % b[5]), by = (int)((i / b[5]) % b[4]), bx = (int)(i / ((size_t)b[5] * b[4]));
        const int gx = wrapi(b[0] + bx, n0), gy = wrapi(b[1] + by, n1), gz = wrapi(b[2] + bz, n2);
        full[(size_t)f * ld + ((size_t)gx * n1 + gy) * n2 + gz] = packed[off[f] + i];
    }
}

/* the kernel variants the tuner chooses from: threads per CTA (a column and its
 * halo hold at most two points per thread) and the CTAs per SM that the
 * registers are limited for */
constexpr int NSHAPE          = 6;
constexpr int SHAPES[NSHAPE]     = { 256, 320, 384, 448, 640, 768 };
constexpr int SHAPE_MINB[NSHAPE] = { 3, 2, 2, 2, 1, 1 };

template <int S> constexpr auto variant() { return &local_step_kernel<SHAPES[S], SHAPE_MINB[S]>; }

/* f<S>() of variant s */
template <template <int> class F, class... A> int with_shape(int s, A... a)
{
    switch (s)
    {
        case 0: return F<0>::run(a...);
        case 1: return F<1>::run(a...);
        case 2: return F<2>::run(a...);
        case 3: return F<3>::run(a...);
        case 4: return F<4>::run(a...);
        default: return F<5>::run(a...);
    }
}

template <int S> struct SetAttr
{
    static int run()
    {
        static bool done = false;
        if (!done)
        {
            MGX_TRY(cuda_check(cudaFuncSetAttribute(variant<S>(),
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)Plane<SHAPES[S]>::SMEM),
                "local smem"));
            done = true;
        }
        return MGX_OK;
    }
};

template <int S> struct Occupancy
{
    static int run()
    {
        if (SetAttr<S>::run() != MGX_OK) return 1;
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, variant<S>(), SHAPES[S],
                Plane<SHAPES[S]>::SMEM)
            != cudaSuccess)
        {
            cudaGetLastError();
            return 1;
        }
        return std::max(n, 1);
    }
};

/* resident CTAs per SM of variant s (also sets its shared-memory limit) */
int max_ctas_per_sm(int s) { return with_shape<Occupancy>(s); }

template <int S> struct Launch
{
    static int run(const StepParams* P, int ctas, cudaStream_t s)
    {
        variant<S>()<<<ctas, SHAPES[S], Plane<SHAPES[S]>::SMEM, s>>>(*P);
        MGX_LAUNCH_CHECK("local_step_kernel");
        return MGX_OK;
    }
};

} // namespace loc
} // namespace mgx

struct mgx_local
{
    mgx_ctx* ctx       = nullptr;
    int nfunc          = 0;
    size_t total       = 0;
    std::vector<int> h_box;      // 6 per orbital
    std::vector<int> h_core;     // 6 per orbital: bounds of the points that a mask reaches
    std::vector<size_t> h_off;   // nfunc + 1
    std::vector<size_t> h_roff;  // nfunc + 1: box columns
    mgx::DeviceBuffer box, off, counter, range, roff;
    // [0]: the cores found at creation; [1]: the whole boxes, for masks that
    // were updated in place since
    mgx::DeviceBuffer core[2];
    mgx::DeviceBuffer items[2][mgx::loc::NSHAPE];
    int nitems[2][mgx::loc::NSHAPE] = {};
    unsigned version[2] = { 0, 0 }; // of masks and corr at creation
    const mgx_masks* masks = nullptr;
    const mgx_masks* corr  = nullptr;
    // chosen configuration
    int shape = 3, ctas_per_sm = 2, use_graph = 1;
    // the captured step, valid for the arguments it was captured with
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph    = nullptr;
    const void* key[5]   = { nullptr, nullptr, nullptr, nullptr, nullptr };
    double key_gamma     = 0.;
    int key_shape = -1, key_ctas = -1;
    unsigned key_version[2] = { 0, 0 };
    ~mgx_local()
    {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};

namespace mgx
{
namespace loc
{
/* the columns of a core of ey x ez for nt threads: as few as hold with the halo
 * in two points per thread, cut into equal parts (the z part rounded up to
 * even, as the threads work on z pairs) */
void fit_columns(int ey, int ez, int nt, int* ty, int* tz)
{
    int best = 1 << 30, area = 0;
    for (int nz = 1; nz <= ez; nz++)
    {
        const int z   = (((ez + nz - 1) / nz) + 1) & ~1;
        const int cap = 2 * nt / (z + 2 * HALO) - 2 * HALO;
        if (cap < 1) continue;
        const int ny = (ey + cap - 1) / cap, y = (ey + ny - 1) / ny;
        const int n  = ((ey + y - 1) / y) * ((ez + z - 1) / z);
        const int a  = (y + 2 * HALO) * (z + 2 * HALO);
        if (n < best || (n == best && a < area))
        {
            best = n;
            area = a;
            *ty  = y;
            *tz  = z;
        }
    }
}

int build_items(mgx_local* L, int whole, int s)
{
    std::vector<int4> it;
    std::vector<std::pair<size_t, int>> order; // largest first
    const int* cores = whole ? nullptr : L->h_core.data();
    auto extent = [&](int f, int k) {
        return cores ? cores[6 * f + 3 + k] - cores[6 * f + k] : L->h_box[6 * f + 3 + k];
    };
    for (int f = 0; f < L->nfunc; f++)
        order.push_back({ (size_t)extent(f, 0) * extent(f, 1) * extent(f, 2), f });
    std::stable_sort(order.begin(), order.end(),
        [](const std::pair<size_t, int>& a, const std::pair<size_t, int>& b) { return a.first > b.first; });
    for (const auto& pr : order)
    {
        if (pr.first == 0) continue;
        const int f = pr.second, ey = extent(f, 1), ez = extent(f, 2);
        const int ya = cores ? cores[6 * f + 1] : 0, za = cores ? cores[6 * f + 2] : 0;
        int ty = 1, tz = 2;
        fit_columns(ey, ez, SHAPES[s], &ty, &tz);
        for (int y = 0; y < ey; y += ty)
            for (int z = 0; z < ez; z += tz)
                it.push_back(make_int4(f, ty | (tz << 16), ya + y, za + z));
    }
    // the points outside the cores last: short items that even out the tail
    if (cores)
        for (const auto& pr : order)
            it.push_back(make_int4(pr.second, 0, 0, 0));
    L->nitems[whole][s] = (int)it.size();
    MGX_TRY(L->items[whole][s].ensure(std::max<size_t>(it.size(), 1) * sizeof(int4)));
    if (!it.empty())
        MGX_TRY(cuda_check(cudaMemcpy(L->items[whole][s].ptr, it.data(), it.size() * sizeof(int4),
                               cudaMemcpyHostToDevice),
            "items upload"));
    return MGX_OK;
}

/* whether the masks changed in place since the cores were found.  The step then
 * marches the whole boxes: 2.92 instead of 1.96 ms for 1536 orbitals on 160^3
 * (3.90 ms with the kernel that always did); a new handle finds the cores again */
int whole_boxes(const mgx_local* L)
{
    return L->masks->version != L->version[0] || L->corr->version != L->version[1];
}

StepParams params(mgx_local* L, int s, const float* psi, const float* phi, const float* V,
    double gamma, float* u, float* w)
{
    StepParams P;
    P.psi   = psi;
    P.phi   = phi;
    P.V     = V;
    P.u     = u;
    P.w     = w;
    P.box   = (const int*)L->box.ptr;
    const int whole = whole_boxes(L);
    P.core  = (const int*)L->core[whole].ptr;
    P.range = whole ? nullptr : (const int*)L->range.ptr;
    P.roff  = (const size_t*)L->roff.ptr;
    P.off   = (const size_t*)L->off.ptr;
    P.mvals = (const float*)L->masks->values[0].ptr;
    P.moff  = (const size_t*)L->masks->offset[0].ptr;
    P.cvals = (const float*)L->corr->values[0].ptr;
    P.coff  = (const size_t*)L->corr->offset[0].ptr;
    P.items   = (const int4*)L->items[whole][s].ptr;
    P.nitems  = L->nitems[whole][s];
    P.counter = (int*)L->counter.ptr;
    const mgx_grid& g = L->ctx->grid;
    for (int i = 0; i < 3; i++)
        P.n[i] = g.n[i];
    const Level L0        = make_level(g, 0);
    const StencilCoeffs c = stencil_coeffs(0, L0.h);
    const double jf = jacobi_factor(0, L0.h);
    auto stencil = [&](double centre, double k) {
        return Stencil19{ (float)(centre + k * c.c0), (float)(k * c.cx[0]), (float)(k * c.cy[0]),
            (float)(k * c.cz[0]), (float)(k * c.cxy), (float)(k * c.cyz), (float)(k * c.cxz) };
    };
    P.lap   = stencil(0., -1.);
    P.sweep = stencil(gamma + jf, -jf * gamma);
    P.A     = stencil(0., 1.);
    P.jf    = (float)jf;
    return P;
}

/* persistent grid of shape s: ctas_per_sm per SM, at most what is resident */
int grid_ctas(mgx_local* L, int s, int ctas_per_sm)
{
    return L->ctx->sm_count * std::max(1, std::min(ctas_per_sm, max_ctas_per_sm(s)));
}

int enqueue(mgx_local* L, int s, int ctas, const StepParams& P, cudaStream_t st)
{
    MGX_TRY(cuda_check(cudaMemsetAsync(L->counter.ptr, 0, sizeof(int), st), "counter reset"));
    return with_shape<Launch>(s, &P, ctas, st);
}

int step(mgx_local* L, const float* psi, const float* phi, const float* V, double gamma, float* u,
    float* w, cudaStream_t st)
{
    const int s         = L->shape;
    const StepParams P  = params(L, s, psi, phi, V, gamma, u, w);
    const int ctas      = grid_ctas(L, s, L->ctas_per_sm);
    if (!L->use_graph) return enqueue(L, s, ctas, P, st);
    const void* key[5] = { psi, phi, V, u, w };
    bool same = L->exec && L->key_gamma == gamma && L->key_shape == s
        && L->key_ctas == L->ctas_per_sm
        && L->key_version[0] == L->masks->version && L->key_version[1] == L->corr->version;
    for (int i = 0; i < 5 && same; i++)
        same = (key[i] == L->key[i]);
    if (!same)
    {
        if (L->exec) cudaGraphExecDestroy(L->exec);
        if (L->graph) cudaGraphDestroy(L->graph);
        L->exec  = nullptr;
        L->graph = nullptr;
        // capture on a private stream (the caller's may be the legacy stream)
        cudaStream_t cs = nullptr;
        MGX_TRY(cuda_check(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "capture stream"));
        // (the kernel's attributes were set by grid_ctas, before the capture)
        int rc = cuda_check(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "begin capture");
        if (rc == MGX_OK)
        {
            const int e1 = enqueue(L, s, ctas, P, cs);
            cudaGraph_t g  = nullptr;
            const int e2   = cuda_check(cudaStreamEndCapture(cs, &g), "end capture");
            rc             = e1 != MGX_OK ? e1 : e2;
            if (rc == MGX_OK)
            {
                rc = cuda_check(cudaGraphInstantiate(&L->exec, g, 0), "graph instantiate");
                L->graph = g;
            }
            else if (g)
                cudaGraphDestroy(g);
        }
        cudaStreamDestroy(cs);
        MGX_TRY(rc);
        for (int i = 0; i < 5; i++)
            L->key[i] = key[i];
        L->key_gamma = gamma;
        L->key_shape = s;
        L->key_ctas  = L->ctas_per_sm;
        L->key_version[0] = L->masks->version;
        L->key_version[1] = L->corr->version;
    }
    count_launch();
    return cuda_check(cudaGraphLaunch(L->exec, st), "graph launch");
}

} // namespace loc
} // namespace mgx

using namespace mgx;

extern "C" {

int mgx_local_create(mgx_ctx* ctx, const mgx_masks* masks, const mgx_masks* corr,
    mgx_local** out)
{
    if (!ctx || !masks || !corr || !out) return fail(MGX_BAD_ARG, "NULL argument");
    if (masks->dtype != MGX_F32 || corr->dtype != MGX_F32)
        return fail(MGX_BAD_ARG, "localized orbitals need FP32 masks");
    if (masks->nfunc != corr->nfunc) return fail(MGX_BAD_ARG, "mask sets of different sizes");
    if (masks->kind != 0 || corr->kind != 1)
        return fail(MGX_BAD_ARG, "orbital masks must clamp (GridMaskMax), correction masks multiply");
    const mgx_grid& g = ctx->grid;
    for (int i = 0; i < 3; i++)
        if (masks->n[i] != g.n[i] || corr->n[i] != g.n[i])
            return fail(MGX_BAD_ARG, "masks of another grid");
    auto L   = std::make_unique<mgx_local>();
    L->ctx   = ctx;
    L->nfunc = masks->nfunc;
    L->masks = masks;
    L->corr  = corr;
    L->h_box.resize(6 * (size_t)L->nfunc);
    L->h_off.resize(L->nfunc + 1);
    size_t tot = 0;
    for (int f = 0; f < L->nfunc; f++)
    {
        if (masks->h_state[0][f] != 2 || corr->h_state[0][f] != 2)
            return fail(MGX_UNSUPPORTED, "orbital %d: mask without a box of values", f);
        for (int k = 0; k < 6; k++)
        {
            const int v = masks->h_box[0][6 * f + k];
            if (corr->h_box[0][6 * f + k] != v)
                return fail(MGX_UNSUPPORTED, "orbital %d: correction box differs from the mask box", f);
            L->h_box[6 * f + k] = v;
        }
        for (int k = 0; k < 3; k++)
            if (L->h_box[6 * f + 3 + k] + 2 * loc::HALO > g.n[k])
                return fail(MGX_UNSUPPORTED, "orbital %d: box wider than the grid less the halo", f);
        L->h_off[f] = tot;
        tot += (size_t)L->h_box[6 * f + 3] * L->h_box[6 * f + 4] * L->h_box[6 * f + 5];
    }
    L->h_off[L->nfunc] = tot;
    L->total           = tot;
    MGX_TRY(L->box.ensure(std::max<size_t>(L->h_box.size(), 1) * sizeof(int)));
    MGX_TRY(L->off.ensure(L->h_off.size() * sizeof(size_t)));
    MGX_TRY(L->counter.ensure(256));
    if (L->nfunc)
    {
        MGX_TRY(cuda_check(cudaMemcpy(L->box.ptr, L->h_box.data(), L->h_box.size() * sizeof(int),
                               cudaMemcpyHostToDevice),
            "box upload"));
        MGX_TRY(cuda_check(cudaMemcpy(L->off.ptr, L->h_off.data(), L->h_off.size() * sizeof(size_t),
                               cudaMemcpyHostToDevice),
            "offset upload"));
    }
    const size_t nf = L->nfunc;
    L->h_roff.assign(nf + 1, 0);
    L->h_core.resize(6 * nf);
    std::vector<int> whole(6 * nf, 0);
    for (size_t f = 0; f < nf; f++)
    {
        const int* e      = &L->h_box[6 * f + 3];
        L->h_roff[f + 1]  = L->h_roff[f] + (size_t)e[1] * e[2];
        for (int k = 0; k < 3; k++)
            whole[6 * f + 3 + k] = e[k];
    }
    L->version[0] = masks->version;
    L->version[1] = corr->version;
    MGX_TRY(L->roff.ensure((nf + 1) * sizeof(size_t)));
    MGX_TRY(L->range.ensure(std::max<size_t>(L->h_roff[nf], 1) * sizeof(int)));
    for (int k = 0; k < 2; k++)
        MGX_TRY(L->core[k].ensure(std::max<size_t>(6 * nf, 1) * sizeof(int)));
    if (nf)
    {
        MGX_TRY(cuda_check(cudaMemcpy(L->roff.ptr, L->h_roff.data(), (nf + 1) * sizeof(size_t),
                               cudaMemcpyHostToDevice),
            "column offset upload"));
        MGX_TRY(cuda_check(cudaMemcpy(L->core[1].ptr, whole.data(), 6 * nf * sizeof(int),
                               cudaMemcpyHostToDevice),
            "box upload"));
        loc::core_kernel<<<(unsigned)nf, 256>>>((const float*)masks->values[0].ptr,
            (const size_t*)masks->offset[0].ptr, (const float*)corr->values[0].ptr,
            (const size_t*)corr->offset[0].ptr, (const int*)L->box.ptr,
            (const size_t*)L->roff.ptr, (int*)L->range.ptr, (int*)L->core[0].ptr);
        MGX_LAUNCH_CHECK("core_kernel");
        MGX_TRY(cuda_check(cudaMemcpy(L->h_core.data(), L->core[0].ptr, 6 * nf * sizeof(int),
                               cudaMemcpyDeviceToHost),
            "cores"));
    }
    for (int s = 0; s < loc::NSHAPE; s++)
        for (int k = 0; k < 2; k++)
            MGX_TRY(loc::build_items(L.get(), k, s));
    *out = L.release();
    return MGX_OK;
}

int mgx_local_destroy(mgx_local* L)
{
    delete L;
    return MGX_OK;
}

int mgx_local_layout(const mgx_local* L, size_t* total, size_t* offsets, int* boxes)
{
    if (!L) return fail(MGX_BAD_ARG, "NULL argument");
    if (total) *total = L->total;
    if (offsets) std::memcpy(offsets, L->h_off.data(), L->h_off.size() * sizeof(size_t));
    if (boxes) std::memcpy(boxes, L->h_box.data(), L->h_box.size() * sizeof(int));
    return MGX_OK;
}

int mgx_local_gather(mgx_local* L, const float* full, size_t ld, float* packed, void* stream)
{
    if (!L || (L->nfunc && (!full || !packed))) return fail(MGX_BAD_ARG, "NULL argument");
    const mgx_grid& g = L->ctx->grid;
    const size_t np   = (size_t)g.n[0] * g.n[1] * g.n[2];
    if (L->nfunc > 1 && ld < np) return fail(MGX_BAD_ARG, "ld %zu < %zu points", ld, np);
    if (L->nfunc == 0) return MGX_OK;
    loc::gather_kernel<<<dim3(64, L->nfunc), 256, 0, (cudaStream_t)stream>>>(full, ld ? ld : np,
        packed, (const int*)L->box.ptr, (const size_t*)L->off.ptr, g.n[0], g.n[1], g.n[2]);
    MGX_LAUNCH_CHECK("gather_kernel");
    return MGX_OK;
}

int mgx_local_scatter(mgx_local* L, const float* packed, float* full, size_t ld, void* stream)
{
    if (!L || (L->nfunc && (!full || !packed))) return fail(MGX_BAD_ARG, "NULL argument");
    const mgx_grid& g = L->ctx->grid;
    const size_t np   = (size_t)g.n[0] * g.n[1] * g.n[2];
    if (L->nfunc > 1 && ld < np) return fail(MGX_BAD_ARG, "ld %zu < %zu points", ld, np);
    if (L->nfunc == 0) return MGX_OK;
    loc::scatter_kernel<<<dim3(64, L->nfunc), 256, 0, (cudaStream_t)stream>>>(packed, full,
        ld ? ld : np, (const int*)L->box.ptr, (const size_t*)L->off.ptr, g.n[0], g.n[1], g.n[2]);
    MGX_LAUNCH_CHECK("scatter_kernel");
    return MGX_OK;
}

int mgx_local_set_config(mgx_local* L, int shape, int ctas_per_sm, int use_graph)
{
    if (!L) return fail(MGX_BAD_ARG, "NULL argument");
    if (shape < 0 || shape >= loc::NSHAPE) return fail(MGX_BAD_ARG, "shape %d", shape);
    if (ctas_per_sm < 1 || ctas_per_sm > 8) return fail(MGX_BAD_ARG, "ctas_per_sm %d", ctas_per_sm);
    L->shape       = shape;
    L->ctas_per_sm = ctas_per_sm;
    L->use_graph   = use_graph ? 1 : 0;
    return MGX_OK;
}

int mgx_local_get_config(const mgx_local* L, int* shape, int* ctas_per_sm, int* use_graph)
{
    if (!L) return fail(MGX_BAD_ARG, "NULL argument");
    if (shape) *shape = L->shape;
    if (ctas_per_sm) *ctas_per_sm = L->ctas_per_sm;
    if (use_graph) *use_graph = L->use_graph;
    return MGX_OK;
}

int mgx_local_step(mgx_local* L, const float* psi, const float* phi, const float* V,
    double gamma, float* u, float* w, void* stream)
{
    if (!L) return fail(MGX_BAD_ARG, "NULL argument");
    if (L->total && (!psi || !phi || !V || !u || !w)) return fail(MGX_BAD_ARG, "NULL block");
    if (u == w || u == psi || u == phi || w == psi || w == phi)
        return fail(MGX_BAD_ARG, "outputs alias the inputs or each other");
    if (L->total == 0) return MGX_OK;
    return loc::step(L, psi, phi, V, gamma, u, w, (cudaStream_t)stream);
}

int mgx_local_tune(mgx_local* L, const float* psi, const float* phi, const float* V,
    double gamma, float* u, float* w, double* ms, int* ncand, void* stream)
{
    if (!L) return fail(MGX_BAD_ARG, "NULL argument");
    if (L->total == 0) return MGX_OK;
    if (!psi || !phi || !V || !u || !w) return fail(MGX_BAD_ARG, "NULL block");
    const cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t e0, e1;
    MGX_TRY(cuda_check(cudaEventCreate(&e0), "event"));
    MGX_TRY(cuda_check(cudaEventCreate(&e1), "event"));
    int best_s = L->shape, best_c = L->ctas_per_sm, k = 0;
    double best = 1e300;
    int rc = MGX_OK;
    for (int s = 0; s < loc::NSHAPE && rc == MGX_OK; s++)
    {
        const int cmax = loc::max_ctas_per_sm(s);
        for (int ci = 0; ci < 4 && rc == MGX_OK; ci++)
        {
            const int c = ci + 1; // 1 to 4 resident CTAs per SM
            double t = 1e300;
            if (c <= cmax)
            {
                const loc::StepParams P = loc::params(L, s, psi, phi, V, gamma, u, w);
                const int ctas          = loc::grid_ctas(L, s, c);
                rc = loc::enqueue(L, s, ctas, P, st); // warm-up
                if (rc == MGX_OK) rc = cuda_check(cudaEventRecord(e0, st), "event");
                for (int r = 0; r < 3 && rc == MGX_OK; r++)
                    rc = loc::enqueue(L, s, ctas, P, st);
                if (rc == MGX_OK) rc = cuda_check(cudaEventRecord(e1, st), "event");
                if (rc == MGX_OK) rc = cuda_check(cudaEventSynchronize(e1), "event");
                float f = 0.f;
                if (rc == MGX_OK) rc = cuda_check(cudaEventElapsedTime(&f, e0, e1), "event");
                t = f / 3.;
                if (t < best)
                {
                    best   = t;
                    best_s = s;
                    best_c = c;
                }
            }
            if (ms && ncand && k < *ncand) ms[k] = t < 1e299 ? t : -1.;
            k++;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    MGX_TRY(rc);
    if (ncand) *ncand = k;
    L->shape       = best_s;
    L->ctas_per_sm = best_c;
    return MGX_OK;
}

} // extern "C"
