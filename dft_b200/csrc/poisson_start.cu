// Start values for the Jacobi Poisson solve (no counterpart in the reference, whose solve
// always starts from zero, HartreePotentialMolecule.cpp:152-155): nested coarse grids, an
// optional network correction (neural.cu) and multigrid V-cycles.  The Jacobi solve that
// follows keeps the reference's stop rule, so every start ends at a Jacobi fixed point to
// the same tolerance; only the number of fine-grid sweeps changes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "common.cuh"
#include "mg_fused.h"
#include "neural.h"
#include "ops.h"

namespace dftb {

int coarse_points(int n) { return std::max(5, (int)std::lround((n - 1) / 2.0) + 1); }

namespace {

// ---------------------------------------------------------------- coarse grid ----------
// Restriction along one axis with the transposed trilinear (hat) weights times h/H, so the
// total charge sum rho dV is kept.  in: (n0, n1, n2) with axis `ax` of length nf; out: the
// same with that axis of length nc.  x_f = lo + f h, X_I = lo + I H.
__global__ void restrict_axis_kernel(const double* __restrict__ in, double* __restrict__ out, int n0, int n1, int n2,
                                     int ax, int nc, double h, double H) {
    int od[3] = {n0, n1, n2};
    const int nf = od[ax];
    od[ax] = nc;
    const long long nout = (long long)od[0] * od[1] * od[2];
    const long long s_in[3] = {1, n0, (long long)n0 * n1};
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nout; q += (long long)gridDim.x * blockDim.x) {
        int idx[3];
        idx[0] = (int)(q % od[0]);
        idx[1] = (int)((q / od[0]) % od[1]);
        idx[2] = (int)(q / ((long long)od[0] * od[1]));
        const int I = idx[ax];
        const double X = I * H;
        const int flo = max(0, (int)ceil((X - H) / h));
        const int fhi = min(nf - 1, (int)floor((X + H) / h));
        long long b = 0;
        for (int d = 0; d < 3; ++d)
            if (d != ax) b += idx[d] * s_in[d];
        double s = 0.0;
        for (int fi = flo; fi <= fhi; ++fi) {
            const double wgt = 1.0 - fabs(fi * h - X) / H;
            if (wgt > 0.0) s += wgt * in[b + fi * s_in[ax]];
        }
        out[q] = s * (h / H);
    }
}

// *s (zeroed before) = bits of max |v|, then 1 if that is zero: the network's input/output scale, kept
// on the device.
__global__ void __launch_bounds__(256) absmax_kernel(long long n, const double* __restrict__ v, double* __restrict__ s) {
    double m = 0.0;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        m = fmax(m, fabs(v[p]));
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0)
        atomicMax(reinterpret_cast<unsigned long long*>(s), (unsigned long long)__double_as_longlong(m));
}
__global__ void one_if_zero_kernel(double* s) {
    if (!(*s > 0.0)) *s = 1.0;
}

__global__ void sum_kernel(long long n, const double* __restrict__ v, double* __restrict__ out) {
    __shared__ double sh[32];
    double m = 0.0;
    for (long long p = threadIdx.x; p < n; p += blockDim.x) m += v[p];
    m = warp_sum(m);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r += sh[w];
        *out = r;
    }
}

struct Gauss {
    double x, y, z, a, inv2w2;
};
__global__ void gauss_density_kernel(Grid g, const Gauss* __restrict__ gs, int k, double* __restrict__ rho) {
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.N; p += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(p % g.nx), j = (int)((p / g.nx) % g.ny), kk = (int)(p / ((long long)g.nx * g.ny));
        const double x = g.xmin + i * g.dx, y = g.ymin + j * g.dy, z = g.zmin + kk * g.dz;
        double s = 0.0;
        for (int q = 0; q < k; ++q) {
            const double dx = x - gs[q].x, dy = y - gs[q].y, dz = z - gs[q].z;
            s += gs[q].a * exp(-(dx * dx + dy * dy + dz * dz) * gs[q].inv2w2);
        }
        rho[p] = s;
    }
}

__global__ void scale_kernel(long long n, double* __restrict__ v, double c) {
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
        v[p] *= c;
}

inline int blocks_for(dft_context* ctx, long long n, int per = 256) {
    const long long b = (n + per - 1) / per;
    return (int)std::max<long long>(1, std::min<long long>(b, (long long)ctx->num_sms * 8));
}

Grid coarse_grid(const Grid& g) {
    dft_grid d{coarse_points(g.nx), coarse_points(g.ny), coarse_points(g.nz), g.xmin, g.xmax, g.ymin,
               g.ymax,          g.zmin,          g.zmax};
    return make_grid(&d);
}

// Nested coarse levels: level 0 = coarse_grid(g), level l+1 = coarse_grid(level l), while
// every axis keeps at least 17 points.  Each level is solved by multigrid cycles from the next
// coarser level's interpolated solution (full multigrid); the finest coarse level's
// solution, interpolated to g, is the start.  Faces are held at zero on every level.  All
// level arrays are carved from one slab of doubles.
struct Level {
    Grid g;
    double *t1, *t2, *rc, *vc;
};

std::vector<Level> plan_levels(const Grid& fine) {
    std::vector<Level> L;
    Grid cur = fine;
    do {
        Level l{};
        l.g = coarse_grid(cur);
        L.push_back(l);
        cur = l.g;
    } while (std::min({cur.nx, cur.ny, cur.nz}) >= 17 && L.size() < 8);
    return L;
}

// separate: with the temporaries of the separate restriction passes
size_t slab_doubles(const Grid& fine, const std::vector<Level>& L, bool separate) {
    size_t n = 8;  // the scale s
    Grid prev = fine;
    for (const Level& l : L) {
        if (separate) n += (size_t)prev.nz * prev.ny * l.g.nx + (size_t)prev.nz * l.g.ny * l.g.nx + 4;
        n += 2 * (size_t)l.g.N + 4;
        // the transfer table between prev and l
        n += 6 * (size_t)(l.g.nx + l.g.ny + l.g.nz) + 2 * (size_t)(prev.nx + prev.ny + prev.nz) + 4;
        prev = l.g;
    }
    return n;
}

// Carves the level arrays and the place of the transfer tables; returns the scale slot.
double* carve(double* slab, const Grid& fine, std::vector<Level>& L, bool separate, double** tables) {
    double* s = slab;
    double* p = slab + 8;
    Grid prev = fine;
    auto take = [&](size_t n) {
        double* q = p;
        p += (n + 1) / 2 * 2;  // keep 16-byte alignment
        return q;
    };
    for (Level& l : L) {
        if (separate) {
            l.t1 = take((size_t)prev.nz * prev.ny * l.g.nx);
            l.t2 = take((size_t)prev.nz * l.g.ny * l.g.nx);
        }
        l.rc = take((size_t)l.g.N);
        l.vc = take((size_t)l.g.N);
        prev = l.g;
    }
    *tables = p;
    return s;
}

void restrict3(dft_context* ctx, const Grid& f, const Grid& c, const double* in, double* t1, double* t2,
               double* out) {
    restrict_axis_kernel<<<blocks_for(ctx, (long long)f.nz * f.ny * c.nx), 256, 0, ctx->stream>>>(
        in, t1, f.nx, f.ny, f.nz, 0, c.nx, f.dx, c.dx);
    restrict_axis_kernel<<<blocks_for(ctx, (long long)f.nz * c.ny * c.nx), 256, 0, ctx->stream>>>(
        t1, t2, c.nx, f.ny, f.nz, 1, c.ny, f.dy, c.dy);
    restrict_axis_kernel<<<blocks_for(ctx, c.N), 256, 0, ctx->stream>>>(t2, out, c.nx, c.ny, f.nz, 2, c.nz, f.dz,
                                                                       c.dz);
    DFT_LAUNCH_CHECK();
    count_launch(ctx, 3);
}

// vup = the nested coarse solution interpolated to g; *s (device) = max |level-0 solution|.
// Returns the multigrid cycles of all coarse levels.
long coarse_solve(dft_context* ctx, double* slab, const Grid& g, const double* rho, double* vup, double** s_out,
                  Grid* gc_out) {
    std::vector<Level> L = plan_levels(g);
    double* tables;
    double* s = carve(slab, g, L, !ctx->mg_fused_restrict, &tables);
    const bool zero = faces_exact(g);  // the coarse boundary follows the fine grid's
    const double* src = rho;
    Grid sg = g;
    std::vector<MGLevel> nest;  // g and the levels, with their transfer tables
    MGLevel m{};
    m.g = g;
    m.ld = g.N;
    nest.push_back(m);
    for (const Level& l : L) {
        m.g = l.g;
        m.ld = l.g.N;
        nest.push_back(m);
    }
    if (ctx->mg_fused_restrict) mg_tables(ctx, nest, tables);
    for (size_t i = 0; i < L.size(); ++i) {
        Level& l = L[i];
        if (ctx->mg_fused_restrict) mg_restrict(ctx, nest[i], l.g, src, l.rc);
        else restrict3(ctx, sg, l.g, src, l.t1, l.t2, l.rc);
        src = l.rc;
        sg = l.g;
    }
    long cycles = 0;
    (void)zero;
    for (int i = (int)L.size() - 1; i >= 0; --i) {
        Level& l = L[i];
        // each level from the next coarser level's interpolated solution (zero on the coarsest)
        if (i + 1 == (int)L.size())
            DFT_CUDA(cudaMemsetAsync(l.vc, 0, sizeof(double) * (size_t)l.g.N, ctx->stream));
        cycles += multigrid(ctx, l.g, l.rc, l.vc, 1e-7, 20, nullptr);
        const Grid& to = i == 0 ? g : L[i - 1].g;
        mg_interpolate(ctx, to, l.g, l.vc, i == 0 ? vup : L[i - 1].vc);
    }
    DFT_CUDA(cudaMemsetAsync(s, 0, sizeof(double), ctx->stream));
    absmax_kernel<<<blocks_for(ctx, L[0].g.N), 256, 0, ctx->stream>>>(L[0].g.N, L[0].vc, s);
    one_if_zero_kernel<<<1, 1, 0, ctx->stream>>>(s);
    DFT_LAUNCH_CHECK();
    count_launch(ctx, 2);
    if (s_out) *s_out = s;
    if (gc_out) *gc_out = L[0].g;
    return cycles;
}

// ---------------------------------------------------------------- multigrid ------------
// Discrete equation per level (faces fixed): den v_p - sum_nb w_d v_nb = src_p, with
// den = 2 (ix2 + iy2 + iz2) and w_d = 1/h_d^2; the fine level's source is 4 pi rho.
__device__ __forceinline__ double nb_sum(const Grid& g, const double* v, long long p) {
    const long long sxy = (long long)g.nx * g.ny;
    return g.ix2 * (v[p - 1] + v[p + 1]) + g.iy2 * (v[p - g.nx] + v[p + g.nx]) + g.iz2 * (v[p - sxy] + v[p + sxy]);
}
__device__ __forceinline__ bool on_face(const Grid& g, long long p) {
    const int i = (int)(p % g.nx), j = (int)((p / g.nx) % g.ny), k = (int)(p / ((long long)g.nx * g.ny));
    return i == 0 || i + 1 == g.nx || j == 0 || j + 1 == g.ny || k == 0 || k + 1 == g.nz;
}

// weighted Jacobi: out = v + omega ((sum + s*src)/den - v); faces copied
__global__ void mg_smooth_kernel(Grid g, const double* __restrict__ src, double sscale, const double* __restrict__ v,
                                 double* __restrict__ out, double omega) {
    const double den = 2.0 * (g.ix2 + g.iy2 + g.iz2);
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.N; p += (long long)gridDim.x * blockDim.x) {
        if (on_face(g, p)) {
            out[p] = v[p];
            continue;
        }
        const double vj = (nb_sum(g, v, p) + sscale * src[p]) / den;
        out[p] = v[p] + omega * (vj - v[p]);
    }
}

// r = s*src - (den v - sum) on the interior, 0 on faces
__global__ void mg_residual_kernel(Grid g, const double* __restrict__ src, double sscale, const double* __restrict__ v,
                                   double* __restrict__ r) {
    const double den = 2.0 * (g.ix2 + g.iy2 + g.iz2);
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.N; p += (long long)gridDim.x * blockDim.x)
        r[p] = on_face(g, p) ? 0.0 : sscale * src[p] - (den * v[p] - nb_sum(g, v, p));
}

// v += trilinear interpolation of the coarse correction e (interior of the fine grid)
__global__ void prolong_add_kernel(Grid f, Grid c, const double* __restrict__ e, double* __restrict__ v) {
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < f.N; p += (long long)gridDim.x * blockDim.x) {
        if (on_face(f, p)) continue;
        const int i = (int)(p % f.nx), j = (int)((p / f.nx) % f.ny), k = (int)(p / ((long long)f.nx * f.ny));
        const double u[3] = {i * f.dx / c.dx, j * f.dy / c.dy, k * f.dz / c.dz};
        const int m[3] = {c.nx, c.ny, c.nz};
        int I[3];
        double w[3];
        for (int d = 0; d < 3; ++d) {
            I[d] = min(max((int)floor(u[d]), 0), m[d] - 2);
            w[d] = fmin(fmax(u[d] - I[d], 0.0), 1.0);
        }
        double s = 0.0;
        for (int t = 0; t < 8; ++t) {
            const int a = t & 1, b = (t >> 1) & 1, cc = t >> 2;
            const double wt = (a ? w[0] : 1.0 - w[0]) * (b ? w[1] : 1.0 - w[1]) * (cc ? w[2] : 1.0 - w[2]);
            s += wt * e[((long long)(I[2] + cc) * c.ny + (I[1] + b)) * c.nx + (I[0] + a)];
        }
        v[p] += s;
    }
}

inline int mg_blocks(dft_context* ctx, long long n) {
    const long long b = (n + 255) / 256;
    return (int)std::max<long long>(1, std::min<long long>(b, (long long)ctx->num_sms * 8));
}


// ---------------------------------------------------------------- multigrid solve ------
// V(2,2) cycles with weighted Jacobi (omega = 0.8) on the nested coarse grids, the same
// charge-conserving restriction and trilinear interpolation, and a coarsest-level red-black
// SOR solve in one block's shared memory (mg_fused.cu).  Faces of every level are held at zero (the boundary of
// every grid whose last nodes land on the bounds).  The "multigrid_fused_restriction" = 0 key takes the
// separate passes below instead.
struct Restriction {
    double *t1, *t2;  // temporaries of the separate restriction passes
};

// Four fields of the finest grid, three of each coarser one; separate: with the passes' temporaries.
size_t mg_doubles(const std::vector<MGLevel>& L, bool separate) {
    size_t n = sizeof(MGHistory) / sizeof(double) + mg_table_doubles(L) + 64 + 4 * ((size_t)L[0].g.N + 32);
    for (size_t i = 0; i < L.size(); ++i) {
        const Grid& g = L[i].g;
        if (i > 0) n += 3 * ((size_t)g.N + 32);
        if (separate && i + 1 < L.size()) {
            const Grid& c = L[i + 1].g;
            n += (size_t)g.nz * g.ny * c.nx + (size_t)g.nz * c.ny * c.nx + 64;
        }
    }
    return n;
}

// One cycle by separate passes below and at level i: v -> v (tmp scratch)
void separate_cycle(dft_context* ctx, std::vector<MGLevel>& L, std::vector<Restriction>& T, size_t i, double sscale,
                    double* v, double* tmp) {
    MGLevel& l = L[i];
    auto smooth = [&](const double* from, double* to) {
        mg_smooth_kernel<<<mg_blocks(ctx, l.g.N), 256, 0, ctx->stream>>>(l.g, l.src, sscale, from, to, 0.8);
        count_launch(ctx);
    };
    smooth(v, tmp);
    smooth(tmp, v);
    mg_residual_kernel<<<mg_blocks(ctx, l.g.N), 256, 0, ctx->stream>>>(l.g, l.src, sscale, v, tmp);
    count_launch(ctx);
    MGLevel& c = L[i + 1];
    restrict3(ctx, l.g, c.g, tmp, T[i].t1, T[i].t2, c.src);
    if (i + 2 == L.size()) {
        mg_coarsest_solve(ctx, c, c.src, ctx->mg_coarsest_sor != 0);
    } else {
        DFT_CUDA(cudaMemsetAsync(c.v, 0, sizeof(double) * (size_t)c.g.N, ctx->stream));
        separate_cycle(ctx, L, T, i + 1, 1.0, c.v, c.tmp);
    }
    prolong_add_kernel<<<mg_blocks(ctx, l.g.N), 256, 0, ctx->stream>>>(l.g, c.g, c.v, v);
    count_launch(ctx);
    smooth(v, tmp);
    smooth(tmp, v);
    DFT_LAUNCH_CHECK();
}

}  // namespace

size_t coarse_slab_doubles(dft_context* ctx, const Grid& g) {
    return slab_doubles(g, plan_levels(g), !ctx->mg_fused_restrict);
}

long coarse_start(dft_context* ctx, double* slab, const Grid& g, const double* rho, double* vup, double** scale_dev) {
    return coarse_solve(ctx, slab, g, rho, vup, scale_dev, nullptr);
}

int multigrid(dft_context* ctx, const Grid& g, const double* rho, double* v, double tol, int max_cycles,
              double* resid_out) {
    std::vector<MGLevel> L = mg_levels(g);
    if (L.back().g.N > MG_COARSEST_MAX) fail(DFT_INVALID_ARGUMENT, "grid too small or too anisotropic for multigrid");
    const bool separate = !ctx->mg_fused_restrict && L.size() > 1;
    double* slab = (double*)ws_get(ctx, WS_PG1, sizeof(double) * mg_doubles(L, separate));
    double* next = slab;
    auto take = [&](size_t n) {
        double* q = next;
        next += (n + 31) / 32 * 32;  // 256-byte alignment
        return q;
    };
    MGHistory* hist = (MGHistory*)take(sizeof(MGHistory) / sizeof(double));
    mg_tables(ctx, L, take(mg_table_doubles(L)));
    // The solve runs on its own copies: the captured cycles below then depend on the grid alone.
    // Cycles alternate between buf[0] and buf[1], so the last two iterates are at hand; v itself, once copied,
    // holds the iterate that a batch of cycles starts from.
    const size_t N = (size_t)g.N, bytes = sizeof(double) * N;
    double* rhs = take(N);
    double* buf[2] = {take(N), take(N)};
    double *tmp = take(N), *saved = v;
    std::vector<Restriction> T(L.size());
    L[0].src = rhs;
    L[0].tmp = tmp;
    for (size_t i = 0; i < L.size(); ++i) {
        if (i > 0) {
            L[i].src = take((size_t)L[i].g.N);
            L[i].v = take((size_t)L[i].g.N);
            L[i].tmp = take((size_t)L[i].g.N);
        }
        if (separate && i + 1 < L.size()) {
            T[i].t1 = take((size_t)L[i].g.nz * L[i].g.ny * L[i + 1].g.nx);
            T[i].t2 = take((size_t)L[i].g.nz * L[i + 1].g.ny * L[i + 1].g.nx);
        }
    }
    DFT_CUDA(cudaMemcpyAsync(rhs, rho, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    DFT_CUDA(cudaMemcpyAsync(buf[0], v, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    DFT_CUDA(cudaMemsetAsync(hist, 0, sizeof(MGHistory), ctx->stream));
    const double den = 2.0 * (g.ix2 + g.iy2 + g.iz2);
    const double fourpi = 4.0 * 3.14159265358979323846;
    const bool sor = ctx->mg_coarsest_sor != 0;
    // one cycle in -> out (in is kept), then the residual's max norm into the history
    auto cycle = [&](const double* in, double* out) {
        if (!separate) {
            L[0].v = out;
            mg_cycle(ctx, L, 0, rhs, nullptr, in, 0, fourpi, nullptr, 1, sor, hist);
        } else {
            mg_start_cycle(ctx, hist);
            DFT_CUDA(cudaMemcpyAsync(out, in, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
            separate_cycle(ctx, L, T, 0, fourpi, out, tmp);
            mg_residual_max(ctx, g, rhs, fourpi, out, hist);
        }
    };
    // The cycle's launch sequence is the same every time for this grid: each direction is captured once
    // as a CUDA graph and replayed.  A capture that fails for any reason leaves the direct launches
    // in place.
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    long long per_replay[2] = {0, 0};
    if (ctx->multigrid_graphs && L.size() > 1) {
        auto bits = [](double x) {
            long long b;
            std::memcpy(&b, &x, sizeof b);
            return b;
        };
        for (int w = 0; w < 2; ++w) {
            const MGGraphKey key{g.nx, g.ny, g.nz, bits(g.dx), bits(g.dy), bits(g.dz), (long long)(uintptr_t)slab, w};
            auto it = ctx->mg_graphs.find(key);
            if (it != ctx->mg_graphs.end()) {
                exec[w] = it->second.exec;
                per_replay[w] = it->second.launches;
                continue;
            }
            const long long l0 = ctx->launches;
            cudaGraph_t graph = nullptr;
            bool captured = false;
            if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                try {
                    cycle(buf[w], buf[1 - w]);
                    captured = true;
                } catch (const Error&) {
                }
                captured = cudaStreamEndCapture(ctx->stream, &graph) == cudaSuccess && graph != nullptr && captured;
            }
            cudaGetLastError();  // a failed capture leaves no sticky error; clear the last one
            per_replay[w] = ctx->launches - l0;
            ctx->launches = l0;
            if (captured && cudaGraphInstantiate(&exec[w], graph, 0) == cudaSuccess) {
                ctx->mg_graphs[key] = {exec[w], per_replay[w]};
            } else {
                exec[w] = nullptr;
                cudaGetLastError();
            }
            if (graph) cudaGraphDestroy(graph);
        }
        // keep a handful: the levels of the current solves (a graph just replayed may still be running)
        if (ctx->mg_graphs.size() > 32) {
            sync(ctx);
            for (auto it = ctx->mg_graphs.begin(); it != ctx->mg_graphs.end() && ctx->mg_graphs.size() > 16;) {
                if (it->second.exec == exec[0] || it->second.exec == exec[1]) {
                    ++it;
                    continue;
                }
                cudaGraphExecDestroy(it->second.exec);
                it = ctx->mg_graphs.erase(it);
            }
        }
    }
    int cur = 0;  // the buffer of the current iterate
    auto run = [&](int m) {
        for (int q = 0; q < m; ++q) {
            if (exec[cur]) {
                DFT_CUDA(cudaGraphLaunch(exec[cur], ctx->stream));
                count_launch(ctx, per_replay[cur]);
            } else {
                cycle(buf[cur], buf[1 - cur]);
            }
            cur = 1 - cur;
        }
    };
    MGHistory* h = (MGHistory*)pinned(ctx, sizeof(MGHistory) / sizeof(double));
    int c = 0;
    double r = 0.0, before = 0.0;
    bool met = false;
    // The count is that of a solve which looks at every cycle's residual.  The residual falls by a
    // steady factor, so after two cycles the ones that cannot be the last yet by that factor are launched together
    // (a host round trip is about 10 us, a cycle at 48^3 about 30); the history then shows the first one
    // that met the tolerance.
    while (c < max_cycles && !met) {
        int m = 1;
        if (c >= 2 && r < before && r > tol && tol > 0.0)
            m = (int)std::max(1.0, std::min(16.0, std::floor(std::log(tol / r) / std::log(r / before))));
        m = std::min(m, max_cycles - c);
        if (m >= 3) DFT_CUDA(cudaMemcpyAsync(saved, buf[cur], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        const int from = cur;
        run(m);
        DFT_CUDA(cudaMemcpyAsync(h, hist, sizeof(MGHistory), cudaMemcpyDeviceToHost, ctx->stream));
        sync(ctx);
        for (int q = 1; q <= m && !met; ++q) {
            before = r;
            std::memcpy(&r, &h->r[(c + q) & 63], sizeof r);
            r /= den;  // the size of the next Jacobi update
            if (!(r < tol)) continue;
            met = true;
            if (q == m - 1) {
                cur = 1 - cur;  // the last cycle was one too many: the iterate before it
            } else if (q < m) {
                DFT_CUDA(cudaMemcpyAsync(buf[from], saved, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
                cur = from;
                run(q);
            }
            m = q;
        }
        c += m;
        // a single level is solved from zero: every further cycle would repeat this one
        if (L.size() == 1) break;
    }
    if (c > 0) DFT_CUDA(cudaMemcpyAsync(v, buf[cur], bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    if (resid_out) *resid_out = r;
    return c;
}

void poisson_start(dft_context* ctx, dft_pnet* net, const Grid& g, const double* rho, double* out, int cycles,
                   PoissonGuessInfo* info) {
    double* slab = (double*)ws_get(ctx, WS_PG0, sizeof(double) * coarse_slab_doubles(ctx, g));
    double* sdev = nullptr;
    const long sw = coarse_start(ctx, slab, g, rho, out, &sdev);
    if (net) pnet_correct(ctx, net, g, rho, out, sdev);
    int used = 0;
    double r = 0.0;
    if (cycles > 0) used = multigrid(ctx, g, rho, out, 0.5e-8, cycles, &r);
    if (info) {
        info->coarse_cycles = sw;
        const Grid gc = coarse_grid(g);
        info->coarse_n[0] = gc.nx;
        info->coarse_n[1] = gc.ny;
        info->coarse_n[2] = gc.nz;
        info->cycles = used;
        info->residual = r;
        double* h = pinned(ctx, 1);
        DFT_CUDA(cudaMemcpyAsync(h, sdev, 8, cudaMemcpyDeviceToHost, ctx->stream));
        sync(ctx);
        info->scale = h[0];
    }
}

int synthetic_density(dft_context* ctx, const Grid& g, unsigned long long seed, int kmin, int kmax, double wmin,
                      double wmax, int ne_min, int ne_max, double* rho) {
    if (kmin < 1 || kmax < kmin || kmax > 64 || wmin <= 0 || wmax < wmin || ne_min < 1 || ne_max < ne_min)
        fail(DFT_INVALID_ARGUMENT, "invalid synthetic density parameters");
    std::mt19937_64 rng(seed);
    std::uniform_int_distribution<int> uk(kmin, kmax), une(ne_min, ne_max);
    std::uniform_real_distribution<double> ux(g.xmin, g.xmax), uy(g.ymin, g.ymax), uz(g.zmin, g.zmax),
        uw(wmin, wmax), ua(0.1, 1.0);
    const int k = uk(rng);
    std::vector<Gauss> gs(k);
    for (auto& q : gs) {
        q.x = ux(rng);
        q.y = uy(rng);
        q.z = uz(rng);
        const double w = uw(rng);
        q.inv2w2 = 1.0 / (2.0 * w * w);
        // amplitude per unit charge of a full Gaussian, times a random weight
        q.a = ua(rng) / std::pow(2.0 * 3.14159265358979323846 * w * w, 1.5);
    }
    const int ne = une(rng);
    Gauss* d = (Gauss*)ws_get(ctx, WS_TMP2, sizeof(Gauss) * gs.size());
    DFT_CUDA(cudaMemcpyAsync(d, gs.data(), sizeof(Gauss) * gs.size(), cudaMemcpyHostToDevice, ctx->stream));
    gauss_density_kernel<<<blocks_for(ctx, g.N), 256, 0, ctx->stream>>>(g, d, k, rho);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    double* tot = (double*)ws_get(ctx, WS_TMP, sizeof(double));
    sum_kernel<<<1, 1024, 0, ctx->stream>>>(g.N, rho, tot);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    double* h = pinned(ctx, 1);
    DFT_CUDA(cudaMemcpyAsync(h, tot, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);  // also keeps gs alive until the density kernel has read it
    const double q = h[0] * g.dV;
    if (!(q > 0.0)) fail(DFT_NUMERICAL, "synthetic density has no charge on the grid");
    scale_kernel<<<blocks_for(ctx, g.N), 256, 0, ctx->stream>>>(g.N, rho, (double)ne / q);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    return ne;
}


}  // namespace dftb
