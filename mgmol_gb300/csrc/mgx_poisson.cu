// pb::Mgm / pb::Vcycle (src/pb/Mgm.h:20-112, src/pb/Vcycle.h:28-249): the
// multigrid Poisson solver on one field, one task, periodic boundaries.
//
// The cycle runs on the stencil engine and the transfer kernels of the
// orbital preconditioner:
//   - a Jacobi sweep is the OP_JACOBI plane kernel (x <- x - jf (A x - f),
//     ping-pong buffers); with jf = 0 the same kernel yields the residual
//     A x - f that Vcycle recomputes after pre-smoothing;
//   - restriction and prolongation-subtraction are restrict_kernel and
//     prolong_kernel (MODE 1);
//   - the residual norms Mgm tests (sqrt(sum r^2 * h^3), GridFunc::norm2,
//     src/pb/GridFunc.cc:2856-2861) are deterministic two-pass device
//     reductions read back once per outer iteration.
// Mgm feeds the cycle the residual rhs - A vh; this implementation passes
// its negative A vh - rhs (the kernel's natural output) and subtracts the
// correction instead of adding it.  Every operation of the cycle is linear
// and commutes exactly with negation, so the iterates are unchanged.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "mgx_internal.cuh"
#include "mgx_stencil.cuh"

namespace mgx
{
int restrict_launch(int, const Level&, const void*, size_t, void*, size_t, int,
    const MaskDev&, cudaStream_t);
int prolong_launch(int, int, const Level&, const void*, size_t, void*, size_t,
    int, const MaskDev&, cudaStream_t);
int scale_launch(int, const void*, size_t, void*, size_t, size_t, int, double, cudaStream_t);

constexpr int NORM_BLOCKS = 512;
// levels of at most so many points are swept without the plane pipeline
constexpr size_t DIRECT_PTS = 16384;

template <typename T>
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const T* __restrict__ u,
    size_t n, double* __restrict__ partial)
{
    __shared__ double red[256];
    double acc = 0.;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
    {
        const double v = (double)u[i];
        acc += v * v;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void __launch_bounds__(256) sum_partials_kernel(const double* __restrict__ partial,
    int n, double* __restrict__ out)
{
    __shared__ double red[256];
    double acc = 0.;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        acc += partial[i];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1)
    {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

/* The part of the cycle below a level of at most BOTTOM_PTS points, in one
 * launch of one CTA: there a sweep's work is under a microsecond, and the ten to
 * twenty launches of its own that each level took (4 to 8 us each) were a tenth
 * of the solve on 96^3.  Every level's fields live in shared memory; the steps
 * are those of PoissonMG::cycle.  LAP: 0 (Laph4M) or 1 (Laph2), on all of these
 * levels. */
constexpr int BOTTOM_PTS    = 512;
constexpr int BOTTOM_LEVELS = 4;

template <typename T>
struct BottomParams
{
    int nlev, nu1, nu2;
    int n[BOTTOM_LEVELS][3];
    T c0[BOTTOM_LEVELS], cf[BOTTOM_LEVELS][3], ce[BOTTOM_LEVELS][3], jf[BOTTOM_LEVELS];
    const T* f; // right-hand side of the first level
    T* x;       // its result
};

template <typename T, int LAP>
__global__ void __launch_bounds__(256) bottom_kernel(const BottomParams<T> p)
{
    // x, x', w and f of every level: 4 (1 + 1/8 + ...) BOTTOM_PTS values
    __shared__ T mem[4 * (BOTTOM_PTS + BOTTOM_PTS / 8 + BOTTOM_PTS / 64 + BOTTOM_PTS / 512)];
    T* base[BOTTOM_LEVELS];
    int np[BOTTOM_LEVELS], cur[BOTTOM_LEVELS];
    {
        T* b = mem;
        for (int l = 0; l < p.nlev; l++)
        {
            np[l]   = p.n[l][0] * p.n[l][1] * p.n[l][2];
            cur[l]  = 0;
            base[l] = b;
            b += 4 * np[l];
        }
    }
    auto X = [&](int l) { return base[l] + cur[l] * np[l]; };
    auto Y = [&](int l) { return base[l] + (1 - cur[l]) * np[l]; };
    auto W = [&](int l) { return base[l] + 2 * np[l]; };
    auto F = [&](int l) { return base[l] + 3 * np[l]; };
    const int tid = threadIdx.x;
    for (int i = tid; i < np[0]; i += 256)
        F(0)[i] = p.f[i];
    __syncthreads();

    // w = A x - f, and x' = x - jf w unless only the residual is wanted
    auto sweep = [&](int l, bool residual) {
        const int ny = p.n[l][1], nz = p.n[l][2], nx = p.n[l][0];
        const T *x = X(l), *f = F(l);
        T *y = Y(l), *w = W(l);
        for (int i = tid; i < np[l]; i += 256)
        {
            const int iz = i % nz, iy = (i / nz) % ny, ix = i / (nz * ny);
            const int zm = iz ? -1 : nz - 1, zp = iz + 1 < nz ? 1 : 1 - nz;
            const int ym = (iy ? -1 : ny - 1) * nz, yp = (iy + 1 < ny ? 1 : 1 - ny) * nz;
            const int xm = (ix ? -1 : nx - 1) * ny * nz, xp = (ix + 1 < nx ? 1 : 1 - nx) * ny * nz;
            const T* q = x + i;
            const T sz = q[zm] + q[zp], sy = q[ym] + q[yp], sx = q[xm] + q[xp];
            T r        = p.c0[l] * q[0] + p.cf[l][2] * sz + p.cf[l][1] * sy + p.cf[l][0] * sx;
            if (LAP == 0)
            {
                r += p.ce[l][0] * (q[xm + zm] + q[xm + zp] + q[xp + zm] + q[xp + zp]); // x z
                r += p.ce[l][1] * (q[ym + zm] + q[ym + zp] + q[yp + zm] + q[yp + zp]); // y z
                r += p.ce[l][2] * (q[xm + ym] + q[xp + ym] + q[xm + yp] + q[xp + yp]); // x y
            }
            r -= f[i];
            if (residual)
                w[i] = r;
            else
                y[i] = q[0] - p.jf[l] * r;
        }
        __syncthreads();
        if (!residual) cur[l] ^= 1;
    };

    for (int l = 0; l < p.nlev; l++)
    {
        // the first sweep from x = 0 is jf f
        for (int i = tid; i < np[l]; i += 256)
            X(l)[i] = p.nu1 > 0 ? p.jf[l] * F(l)[i] : (T)0;
        __syncthreads();
        for (int s = 1; s < p.nu1; s++)
            sweep(l, false);
        if (l + 1 == p.nlev) break;
        sweep(l, true);
        // full weighting (restrict_kernel)
        const int nx = p.n[l][0], ny = p.n[l][1], nz = p.n[l][2];
        const int cy = ny >> 1, cz = nz >> 1;
        const T* w = W(l);
        for (int i = tid; i < np[l + 1]; i += 256)
        {
            const int iz = 2 * (i % cz), iy = 2 * ((i / cz) % cy), ix = 2 * (i / (cz * cy));
            const int zm = iz ? -1 : nz - 1, zp = 1;
            const int ym = (iy ? -1 : ny - 1) * nz, yp = nz;
            const int xm = (ix ? -1 : nx - 1) * ny * nz, xp = ny * nz;
            const T* q = w + (ix * ny + iy) * nz + iz;
            const T face   = q[xp] + q[xm] + q[yp] + q[ym] + q[zm] + q[zp];
            const T corner = q[xp + yp + zm] + q[xp + yp + zp] + q[xp + ym + zm] + q[xp + ym + zp]
                             + q[xm + yp + zm] + q[xm + yp + zp] + q[xm + ym + zm] + q[xm + ym + zp];
            const T edge   = q[yp + zm] + q[yp + zp] + q[ym + zm] + q[ym + zp] + q[xp + zm]
                           + q[xp + zp] + q[xm + zm] + q[xm + zp] + q[xm + ym] + q[xp + ym]
                           + q[xm + yp] + q[xp + yp];
            F(l + 1)[i] = (T)(1. / 64.) * ((T)8. * q[0] + (T)4. * face + (T)2. * edge + corner);
        }
        __syncthreads();
    }
    for (int l = p.nlev - 1; l >= 0; l--)
    {
        if (l + 1 < p.nlev)
        {
            // x -= trilinear interpolation of the level below (prolong_kernel)
            const int ny = p.n[l][1], nz = p.n[l][2];
            const int cx = p.n[l][0] >> 1, cy = ny >> 1, cz = nz >> 1;
            const T* e = X(l + 1);
            T* x       = X(l);
            for (int i = tid; i < np[l]; i += 256)
            {
                const int iz = i % nz, iy = (i / nz) % ny, ix = i / (nz * ny);
                const int az = iz & 1, ay = iy & 1, ax = ix & 1;
                const int jz = iz >> 1, jy = iy >> 1, jx = ix >> 1;
                const int dz = az ? (jz + 1 < cz ? 1 : 1 - cz) : 0;
                const int dy = ay ? (jy + 1 < cy ? 1 : 1 - cy) * cz : 0;
                const int dx = ax ? (jx + 1 < cx ? 1 : 1 - cx) * cy * cz : 0;
                const T* q   = e + (jx * cy + jy) * cz + jz;
                // every odd direction halves a sum of two
                T v = q[0];
                if (az) v = v + q[dz];
                if (ay) v = v + (az ? q[dy] + q[dy + dz] : q[dy]);
                if (ax)
                {
                    T u = q[dx];
                    if (az) u = u + q[dx + dz];
                    if (ay) u = u + (az ? q[dx + dy] + q[dx + dy + dz] : q[dx + dy]);
                    v = v + u;
                }
                x[i] -= v * (T)(1. / (1 << (ax + ay + az)));
            }
            __syncthreads();
        }
        for (int s = 0; s < p.nu2; s++)
            sweep(l, false);
    }
    const T* x = X(0);
    for (int i = tid; i < np[0]; i += 256)
        p.x[i] = x[i];
}

namespace
{
struct PoissonMG
{
    int dtype;
    int nu1, nu2;
    cudaStream_t s;
    std::vector<Level> lev;
    std::vector<int> op;      // operator per level
    std::vector<double> jf;   // Jacobi factor per level
    std::vector<void*> x0, x1, w, f;
    void* partial = nullptr;  // NORM_BLOCKS doubles + the result
    int* err      = nullptr;
    size_t es     = 8;

    // one Jacobi sweep; gamma: from gamma f[l] instead of u
    int sweep(int l, const void* u, void* out, void* wout, double factor, double gamma = 0.)
    {
        PlaneParams p;
        p.u   = u;
        p.ldu = lev[l].npts();
        p.f   = f[l];
        p.ldf = lev[l].npts();
        p.out = out;
        p.ldo = lev[l].npts();
        p.w   = wout;
        p.ldw = lev[l].npts();
        for (int i = 0; i < 3; i++)
            p.n[i] = lev[l].n[i];
        p.err      = err;
        p.gamma_in = gamma;
        // small levels: the kernel without a plane pipeline starts sooner (4
        // against 8 us a sweep at 12^3 and 24^3)
        return stencil_launch(OP_JACOBI, op[l], dtype, dtype, p, lev[l], factor, 1, s,
            lev[l].npts() <= DIRECT_PTS ? 1 : 0);
    }

    // the cycle from level l down in bottom_kernel; MGX_UNSUPPORTED where it
    // cannot run.  The result goes to x0[l].
    int bottom(int l)
    {
        const int nl = (int)lev.size() - l;
        if (nl > BOTTOM_LEVELS || lev[l].npts() > BOTTOM_PTS || op[l] > 1) return MGX_UNSUPPORTED;
        for (int k = l; k < (int)lev.size(); k++)
            if (op[k] != op[l]) return MGX_UNSUPPORTED;
        return dtype == MGX_F64 ? bottom_t<double>(l, nl) : bottom_t<float>(l, nl);
    }

    template <typename T>
    int bottom_t(int l, int nl)
    {
        BottomParams<T> p;
        p.nlev = nl;
        p.nu1  = nu1;
        p.nu2  = nu2;
        for (int k = 0; k < nl; k++)
        {
            const Level& L        = lev[l + k];
            const StencilCoeffs c = stencil_coeffs(op[l], L.h);
            for (int i = 0; i < 3; i++)
                p.n[k][i] = L.n[i];
            p.c0[k]    = (T)c.c0;
            p.cf[k][0] = (T)c.cx[0];
            p.cf[k][1] = (T)c.cy[0];
            p.cf[k][2] = (T)c.cz[0];
            p.ce[k][0] = (T)c.cxz;
            p.ce[k][1] = (T)c.cyz;
            p.ce[k][2] = (T)c.cxy;
            p.jf[k]    = (T)jf[l + k];
        }
        p.f = (const T*)f[l];
        p.x = (T*)x0[l];
        if (op[l] == 0)
            bottom_kernel<T, 0><<<1, 256, 0, s>>>(p);
        else
            bottom_kernel<T, 1><<<1, 256, 0, s>>>(p);
        MGX_LAUNCH_CHECK("bottom_kernel");
        return MGX_OK;
    }

    // Vcycle at level l from x = 0; returns the buffer (0: x0, 1: x1) that
    // holds the result, or a negative status
    int cycle(int l)
    {
        int st = bottom(l);
        if (st == MGX_OK) return 0;
        if (st != MGX_UNSUPPORTED) return -st - 1;
        int cur      = 0;
        auto X       = [&](int b) { return b ? x1[l] : x0[l]; };
        const size_t np = lev[l].npts();
        // the first sweep from x = 0 is x = jf f, and the second one reads f
        // times jf where its kernel can
        int done = std::min(nu1, 1);
        if (nu1 >= 2)
        {
            st = sweep(l, f[l], x1[l], nullptr, jf[l], jf[l]);
            if (st == MGX_OK)
            {
                done = 2;
                cur  = 1;
            }
            else if (st != MGX_UNSUPPORTED)
                return -st - 1;
        }
        if (done == 0)
            st = cuda_check(cudaMemsetAsync(x0[l], 0, np * es, s), "mgm zero");
        else if (done == 1)
            st = scale_launch(dtype, f[l], np, x0[l], np, np, 1, jf[l], s);
        if (st != MGX_OK) return -st - 1;
        for (int i = done; i < nu1; i++)
        {
            st = sweep(l, X(cur), X(cur ^ 1), nullptr, jf[l]);
            if (st != MGX_OK) return -st - 1;
            cur ^= 1;
        }
        if (l + 1 < (int)lev.size())
        {
            // res = A x - rhs (src/pb/Vcycle.h:165-167): a sweep with factor 0
            // copies x to the other buffer and writes the residual to w
            st = sweep(l, X(cur), X(cur ^ 1), w[l], 0.);
            if (st != MGX_OK) return -st - 1;
            st = restrict_launch(dtype, lev[l], w[l], lev[l].npts(), f[l + 1],
                lev[l + 1].npts(), 1, MaskDev(), s);
            if (st != MGX_OK) return -st - 1;
            const int c = cycle(l + 1);
            if (c < 0) return c;
            // x -= extend(ucoarse) (src/pb/Vcycle.h:197-198)
            st = prolong_launch(dtype, 1, lev[l], c ? x1[l + 1] : x0[l + 1],
                lev[l + 1].npts(), X(cur), lev[l].npts(), 1, MaskDev(), s);
            if (st != MGX_OK) return -st - 1;
        }
        for (int i = 0; i < nu2; i++)
        {
            st = sweep(l, X(cur), X(cur ^ 1), nullptr, jf[l]);
            if (st != MGX_OK) return -st - 1;
            cur ^= 1;
        }
        return cur;
    }

    int norm(const void* u, size_t n, double vel, double* out)
    {
        double* part = (double*)partial;
        if (dtype == MGX_F64)
            sumsq_partial_kernel<double><<<NORM_BLOCKS, 256, 0, s>>>((const double*)u, n, part);
        else
            sumsq_partial_kernel<float><<<NORM_BLOCKS, 256, 0, s>>>((const float*)u, n, part);
        MGX_LAUNCH_CHECK("sumsq_partial_kernel");
        sum_partials_kernel<<<1, 256, 0, s>>>(part, NORM_BLOCKS, part + NORM_BLOCKS);
        MGX_LAUNCH_CHECK("sum_partials_kernel");
        double h = 0.;
        MGX_TRY(cuda_check(cudaMemcpyAsync(&h, part + NORM_BLOCKS, sizeof(double),
                               cudaMemcpyDeviceToHost, s),
            "norm read-back"));
        MGX_TRY(cuda_check(cudaStreamSynchronize(s), "norm sync"));
        *out = std::sqrt(h * vel);
        return MGX_OK;
    }
};
} // namespace

int mgm_solve(mgx_ctx* ctx, const mgx_mgm_params* P, int dtype, void* vh,
    const void* rho, mgx_mgm_result* R, cudaStream_t s)
{
    if (!P || !vh || !rho || !R) return fail(MGX_BAD_ARG, "mgm: null argument");
    if (vh == rho) return fail(MGX_BAD_ARG, "mgm: vh and rho alias");
    const int radius = lap_radius(P->lap_type);
    if (radius < 0) return fail(MGX_BAD_ARG, "lap_type %d", P->lap_type);
    if (P->nu1 < 0 || P->nu2 < 0 || P->max_sweeps < 0 || P->max_levels < 0)
        return fail(MGX_BAD_ARG, "mgm: negative count");
    const int g0 = P->ghosts > 0 ? P->ghosts : radius;
    if (g0 < radius) return fail(MGX_BAD_ARG, "ghost width %d below operator radius %d", g0, radius);

    PoissonMG M;
    M.dtype = dtype;
    M.nu1   = P->nu1;
    M.nu2   = P->nu2;
    M.s     = s;
    M.es    = dtype_size(dtype);
    // levels: coarsen while every dimension is even and at least twice the
    // ghost width of the level's function, at most max_levels times
    // (src/pb/Vcycle.h:52-60,154-188).  Each coarse level takes the lower-
    // order operator (Laph4M stays Laph4M; Laph8 -> Laph6 -> Laph4 -> Laph2,
    // src/pb/Laph8.h:79-87, Laph6.h:79-87, Laph4.h:75-83), whose grid has
    // that operator's minimum ghost width; the coarse function's ghost width
    // is max(ghosts of the finer operator's grid - 1, 1) (Vcycle.h:176-180),
    // with the caller's g0 on the fine level.
    static const int lower[5] = { 0, 1, 1, 2, 3 };
    int o = P->lap_type, ng = g0, op_ng = g0;
    for (int l = 0;; l++)
    {
        const Level L = make_level(ctx->grid, l);
        M.lev.push_back(L);
        M.op.push_back(o);
        M.jf.push_back(jacobi_factor(o, L.h));
        bool coarsen = (l < P->max_levels);
        for (int i = 0; i < 3; i++)
            if ((L.n[i] & 1) || L.n[i] < 2 * ng) coarsen = false;
        if (!coarsen) break;
        ng    = std::max(op_ng - 1, 1);
        o     = lower[o];
        op_ng = lap_radius(o);
    }
    const int nl = (int)M.lev.size();
    // workspace: per level x0, x1, w, f (the fine level's f holds the outer
    // residual), then rhs, a scratch copy of vh and the norm partials
    size_t total = 0;
    std::vector<size_t> off;
    auto take = [&](size_t bytes) {
        off.push_back(total);
        total += ((bytes + 255) / 256) * 256;
    };
    for (int l = 0; l < nl; l++)
        for (int k = 0; k < 4; k++)
            take(M.lev[l].npts() * M.es);
    take(M.lev[0].npts() * M.es); // rhs
    take(M.lev[0].npts() * M.es); // scratch copy of vh
    take((NORM_BLOCKS + 1) * sizeof(double));
    MGX_TRY(ctx->mgm.ensure(total));
    MGX_TRY(ctx->flag.ensure(16));
    char* base = (char*)ctx->mgm.ptr;
    for (int l = 0; l < nl; l++)
    {
        M.x0.push_back(base + off[4 * l + 0]);
        M.x1.push_back(base + off[4 * l + 1]);
        M.w.push_back(base + off[4 * l + 2]);
        M.f.push_back(base + off[4 * l + 3]);
    }
    void* rhs     = base + off[4 * nl];
    void* scratch = base + off[4 * nl + 1];
    M.partial     = base + off[4 * nl + 2];
    M.err         = (int*)ctx->flag.ptr;
    MGX_TRY(cuda_check(cudaMemsetAsync(M.err, 0, sizeof(int), s), "flag reset"));

    const Level& F  = M.lev[0];
    const size_t np = F.npts();
    const double vel = F.h[0] * F.h[1] * F.h[2];
    // rhs = A.rhs(rho): B rho for Mehrstellen, rho otherwise (src/pb/Mgm.h:36-41)
    if (P->lap_type == 0)
    {
        PlaneParams p;
        p.u   = rho;
        p.ldu = np;
        p.out = rhs;
        p.ldo = np;
        for (int i = 0; i < 3; i++)
            p.n[i] = F.n[i];
        MGX_TRY(stencil_launch(OP_RHS, 0, dtype, dtype, p, F, 0., 1, s));
    }
    else
        MGX_TRY(cuda_check(cudaMemcpyAsync(rhs, rho, np * M.es, cudaMemcpyDeviceToDevice, s),
            "rhs copy"));
    double rhs_norm = 0.;
    MGX_TRY(M.norm(rhs, np, vel, &rhs_norm));
    const double inv_rhs_norm = 1. / rhs_norm;

    // the outer residual A vh - rhs goes to r via a factor-0 sweep on the
    // fine level against rhs (its x output is a scratch copy); r is then the
    // fine-level right-hand side of the cycle
    void* r = M.f[0];
    auto residual = [&]() -> int {
        M.f[0] = rhs;
        const int st = M.sweep(0, vh, scratch, r, 0.);
        M.f[0] = r;
        return st;
    };
    double init = 1., res_norm = 0.;
    bool converged = false;
    int sweeps     = 0;
    R->final_residual = R->final_relative_residual = 0.;
    for (int i = 0; i < P->max_sweeps; i++)
    {
        MGX_TRY(residual());
        MGX_TRY(M.norm(r, np, vel, &res_norm));
        if (i == 0) init = res_norm;
        if (res_norm * inv_rhs_norm < P->tol)
        {
            R->final_residual          = res_norm;
            R->final_relative_residual = res_norm * inv_rhs_norm;
            converged                  = true;
            break;
        }
        const int c = M.cycle(0);
        if (c < 0) return -c - 1;
        sweeps++;
        // vh += work1, with work1 the cycle of the negated residual
        MGX_TRY(mgx_axpy(np, -1., (mgx_dtype)dtype, c ? M.x1[0] : M.x0[0], vh, s));
    }
    if (!converged)
    {
        MGX_TRY(residual());
        MGX_TRY(M.norm(r, np, vel, &res_norm));
        R->final_residual          = res_norm;
        R->final_relative_residual = res_norm * inv_rhs_norm;
    }
    int herr = 0;
    MGX_TRY(cuda_check(cudaMemcpyAsync(&herr, M.err, sizeof(int), cudaMemcpyDeviceToHost, s),
        "flag read-back"));
    MGX_TRY(cuda_check(cudaStreamSynchronize(s), "mgm sync"));
    if (herr) return fail(MGX_TIMEOUT, "stencil pipeline wait gave up");
    R->residual_reduction = R->final_residual / init;
    R->nb_sweeps          = sweeps;
    R->converged          = converged ? 1 : 0;
    R->levels             = nl;
    return MGX_OK;
}
} // namespace mgx
