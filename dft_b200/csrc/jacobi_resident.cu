// Jacobi Poisson solve in one cooperative launch with the grid resident in shared memory (cubes up to
// 86^3), T sweeps per exchange between blocks.
//
// The sweep of a small grid is a fraction of a microsecond of work, so what bounds a solve of
// thousands of sweeps is the exchange between SMs.  Every block owns a box of interior points and keeps it, a
// T-point halo and 4 pi rho in shared memory.  A round is T sweeps, each on a box one point smaller
// per side than the last (the halo is recomputed redundantly); then the owned points go out and the
// halo comes in.  Measured on B200: a grid barrier with its two fences is 3,100 cycles and the fetch
// behind it another 500 to 1,000, so there is no barrier: a value travels as two 8-byte words, each
// 4 bytes of it and the round's number, and the reader polls the words themselves (1,900 cycles from
// store to use across the dies, fences and atomics included in neither).
//
// The stop rule asks whether any block saw |V' - V| >= tol.  Each block posts one bit per sweep of a
// round on a board in the same form; everyone reads the board of round q while computing round q + 2, when
// it has long arrived, and takes the same decision at the same point.  The owned points of the last
// four rounds are still in the exchange ring then, so the stopping round is redone from its start up to
// the stopping sweep, which also gives the maximum to report.  Values and sweep count are those of
// the one-sweep kernel, bit for bit: same operations in the same order, the division through
// exact_div.cuh.
//
// A half warp sweeps one row (two rows of at most 16 points are two shared-memory wavefronts whatever
// their pitch); shared-memory reads, 7 per point, are what bounds a sweep.
//
// 48^3 to the stop rule (T = 3): 1.44 us per sweep; 6.46 for the 16-block cluster that exchanged whole planes
// every sweep, 3.57 for this layout behind a grid barrier, 7.6 to 8.3 for one launch per sweep.
//
// Every wait is bounded: a thread that polls poll_limit times, or sees the error word set,
// sets it and its block returns; the host reports it.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "exact_div.cuh"
#include "ops.h"
#include "xc_device.cuh"

namespace dftb {

namespace {

constexpr int RJ_THREADS = 512;
constexpr int RJ_ROWS = RJ_THREADS / 16;
constexpr int RJ_TMAX = 4;
constexpr int RJ_HALO = 8;                   // halo points per thread, at most
constexpr size_t RJ_SMEM = 200 * 1024;       // beside the static arrays
constexpr int RJ_DELAY = 2;                  // rounds between a round and the reading of its board
constexpr int RJ_RING = RJ_DELAY + 2;        // exchange slots: the rounds a block may still go back to
constexpr int RJ_BOARDS = 2 * RJ_DELAY + 2;  // who posts round r has seen every board of r - 3, so none older than r - 5 is read

struct JacobiRCtrl {
    int error;
    int in_buf1;  // the result is in buf1
    long long sweeps;
    unsigned long long last_diff;  // bits of a non-negative double
};

struct RJShape {
    int bx, by, bz;  // blocks per axis
    int points;      // most region points of a block
};

// A double in two words that carry the round's number beside their half of it.
struct Packet {
    unsigned long long lo, hi;
};
__device__ __forceinline__ void post(Packet* p, double v, unsigned tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
    const unsigned long long lo = (b & 0xffffffffULL) | t, hi = (b >> 32) | t;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ Packet look(const Packet* p) {
    Packet q;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(q.lo), "=l"(q.hi) : "l"(p) : "memory");
    return q;
}
__device__ __forceinline__ bool has(const Packet& q, unsigned tag) {
    return (unsigned)(q.lo >> 32) == tag && (unsigned)(q.hi >> 32) == tag;
}
__device__ __forceinline__ double value(const Packet& q) {
    return __longlong_as_double((long long)((q.lo & 0xffffffffULL) | (q.hi << 32)));
}

// interior points of axis length n owned by part i of m: [begin(i), begin(i + 1)) in grid indices
__host__ __device__ __forceinline__ int part_begin(int n, int i, int m) {
    return 1 + (int)(((long long)(n - 2) * i) / m);
}

template <int T>
__global__ void __launch_bounds__(RJ_THREADS, 1)
    jacobi_resident_kernel(Grid g, const double* __restrict__ rho, double* buf0, double* buf1, Packet* ring,
                           Packet* board, JacobiRCtrl* ctrl, ExactDiv dv, double tol, long long cap, RJShape sh,
                           long long poll_limit) {
    extern __shared__ double sm[];
    __shared__ unsigned s_mine[2];  // bit t - 1: this block has |dV| >= tol in sweep t of the round
    __shared__ unsigned s_over[2];  // the same over all blocks, for the round whose board was read last
    __shared__ int s_fail, s_halo;
    double* S0 = sm;
    double* S1 = sm + sh.points;
    double* R = sm + 2 * sh.points;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, ix = b % sh.bx, iy = (b / sh.bx) % sh.by, iz = b / (sh.bx * sh.by);
    // owned box and region (owned + T, clipped to the grid)
    const int x0 = part_begin(g.nx, ix, sh.bx), x1 = part_begin(g.nx, ix + 1, sh.bx);
    const int y0 = part_begin(g.ny, iy, sh.by), y1 = part_begin(g.ny, iy + 1, sh.by);
    const int z0 = part_begin(g.nz, iz, sh.bz), z1 = part_begin(g.nz, iz + 1, sh.bz);
    const int lx = max(0, x0 - T), hx = min(g.nx, x1 + T);
    const int ly = max(0, y0 - T), hy = min(g.ny, y1 + T);
    const int lz = max(0, z0 - T), hz = min(g.nz, z1 + T);
    const int ex = hx - lx, ey = hy - ly, ez = hz - lz, exy = ex * ey;
    const int sxy = g.nx * g.ny;
    const double c4pi = 4.0 * xcf::PI;
    auto global_index = [&](int li) {
        const int z = li / exy, r = li - z * exy, y = r / ex;
        return (lz + z) * sxy + (ly + y) * g.nx + lx + (r - y * ex);
    };

    // ---- halo list: the points of other blocks (not the faces, which never change) within T steps
    // of the owned box, in region order; S1 holds it until every thread has taken its entries
    int* list = reinterpret_cast<int*>(S1);
    if (tid == 0) s_halo = s_fail = 0, s_over[0] = s_over[1] = s_mine[0] = s_mine[1] = 0;
    __syncthreads();
    for (int i0 = warp * 32; i0 < exy * ez; i0 += RJ_THREADS) {
        const int i = i0 + lane;
        bool want = false;
        if (i < exy * ez) {
            const int zz = i / exy, r = i - zz * exy, yy = r / ex;
            const int x = lx + r - yy * ex, y = ly + yy, z = lz + zz;
            const int dist = max(max(x0 - x, x - (x1 - 1)), 0) + max(max(y0 - y, y - (y1 - 1)), 0) +
                             max(max(z0 - z, z - (z1 - 1)), 0);
            const bool face = x == 0 || x == g.nx - 1 || y == 0 || y == g.ny - 1 || z == 0 || z == g.nz - 1;
            want = dist > 0 && dist <= T && !face;
        }
        const unsigned m = __ballot_sync(0xffffffffu, want);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&s_halo, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1));
        if (want && at < RJ_HALO * RJ_THREADS) list[at] = i;
    }
    __syncthreads();
    const int nhalo = min(s_halo, RJ_HALO * RJ_THREADS);
    int hl[RJ_HALO], hg[RJ_HALO];  // region and grid index of this thread's halo points
#pragma unroll
    for (int q = 0; q < RJ_HALO; ++q) {
        hl[q] = tid + q * RJ_THREADS < nhalo ? list[tid + q * RJ_THREADS] : -1;
        hg[q] = hl[q] >= 0 ? global_index(hl[q]) : 0;
    }
    __syncthreads();

    // ---- a thread's points of sweep t of tsw: a run of n points along z from region index li; those at
    // [o0, o1) of the run are owned
    struct Run {
        int li, n, o0, o1;
    };
    auto run_of = [&](int t, int tsw) -> Run {
        const int e = tsw - t;
        const int ax = max(1, x0 - e), bx = min(g.nx - 1, x1 + e);
        const int ay = max(1, y0 - e), by = min(g.ny - 1, y1 + e);
        const int az = max(1, z0 - e), bz = min(g.nz - 1, z1 + e);
        // a half warp per row of at most 16 points, the rows cut along z so that the half warps
        // share them evenly (at most RJ_ROWS rows)
        const int xs = (bx - ax + 15) / 16, rows = xs * (by - ay), d = bz - az;
        const int len = (d + RJ_ROWS / rows - 1) / (RJ_ROWS / rows);
        const int hw = tid >> 4, sg = hw / rows, c = hw - sg * rows, cy = c / xs;
        const int x = ax + (c - cy * xs) * 16 + (tid & 15), y = ay + cy, zb = az + sg * len;
        Run r;
        r.n = x < bx ? max(0, min(len, bz - zb)) : 0;
        r.li = r.n ? (zb - lz) * exy + (y - ly) * ex + (x - lx) : exy;
        const bool own = x >= x0 && x < x1 && y >= y0 && y < y1;
        r.o0 = own ? z0 - zb : 0;
        r.o1 = own ? z1 - zb : 0;
        return r;
    };
    // the new value of region point li (between `below` and `above` along z), unrounded range check in bad
    auto update = [&](const double* cur, int li, double below, double above, double& acc, bool& bad) -> double {
        const double sx = __dadd_rn(cur[li - 1], cur[li + 1]);
        const double sy = __dadd_rn(cur[li - ex], cur[li + ex]);
        const double sz = __dadd_rn(below, above);
        acc = __dadd_rn(__dmul_rn(g.ix2, sx), __dmul_rn(g.iy2, sy));
        acc = __dadd_rn(acc, __dmul_rn(g.iz2, sz));
        acc = __dadd_rn(acc, R[li]);
        return divide_fast(acc, dv, bad);
    };
    // one sweep over this thread's run, two points at a time; where `out` is given the new values are
    // posted there (out: the packet of the run's first point)
    auto sweep = [&](const double* cur, double* nxt, const Run& u, Packet* out, unsigned tag) -> double {
        double md = 0.0;  // max |dV| of this thread's owned points
        int li = u.li;
        double below = cur[li - exy], c = cur[li];
        for (int i = 0; i < u.n; i += 2, li += 2 * exy) {
            const bool two = i + 1 < u.n;
            const int l2 = two ? li + exy : li;
            const double c2 = cur[li + exy];
            const double above2 = cur[l2 + exy];
            double a1, a2;
            bool bad1, bad2;
            double v1 = update(cur, li, below, c2, a1, bad1);
            double v2 = update(cur, l2, c, above2, a2, bad2);
            if (bad1 || bad2 || dv.general) {
                v1 = divide(a1, dv);
                v2 = divide(a2, dv);
            }
            nxt[li] = v1;
            if (i >= u.o0 && i < u.o1) md = fmax(md, fabs(v1 - c));
            if (out) post(out + (long long)i * sxy, v1, tag);
            if (two) {
                nxt[l2] = v2;
                if (i + 1 >= u.o0 && i + 1 < u.o1) md = fmax(md, fabs(v2 - c2));
                if (out) post(out + (long long)(i + 1) * sxy, v2, tag);
            }
            below = c2;
            c = above2;
        }
        return md;
    };

    // ---- start: the whole region, and the faces in both buffers
    for (int i = tid; i < exy * ez; i += RJ_THREADS) {
        const int gi = global_index(i);
        const double v = __ldcg(buf0 + gi);
        S0[i] = v;
        S1[i] = v;
        R[i] = __dmul_rn(c4pi, __ldg(rho + gi));
    }
    Run runs[T];
#pragma unroll
    for (int t = 0; t < T; ++t) runs[t] = run_of(t + 1, T);
    const int out_gi = global_index(runs[T - 1].li);
    double *cur = S0, *nxt = S1;
    __syncthreads();
    for (long long round = 0;; ++round) {
        if (round > 0) {
            // ---- halo of this round
            const Packet* slot = ring + (round % RJ_RING) * g.N;
            const unsigned tag = (unsigned)round;
            Packet p[RJ_HALO];
#pragma unroll
            for (int q = 0; q < RJ_HALO; ++q)
                if (hl[q] >= 0) p[q] = look(slot + hg[q]);
            long long polls = 0;
#pragma unroll
            for (int q = 0; q < RJ_HALO; ++q) {
                if (hl[q] < 0) continue;
                while (!has(p[q], tag)) {
                    if (++polls >= poll_limit || ((polls & 1023) == 0 && atomicAdd(&ctrl->error, 0) != 0)) {
                        atomicExch(&ctrl->error, 1);
                        s_fail = 1;
                        break;
                    }
                    p[q] = look(slot + hg[q]);
                }
                cur[hl[q]] = value(p[q]);
            }
            __syncthreads();
            if (s_fail) return;
            // ---- the decision on round `past`, whose board was read during the last round
            const long long past = round - 1 - RJ_DELAY;
            if (past >= 0) {
                const unsigned over = s_over[(round - 1) & 1];
                int fin = 0;
#pragma unroll
                for (int t = 1; t <= T; ++t)
                    if (!fin && ((tol > 0.0 && !(over >> (t - 1) & 1)) || past * T + t >= cap)) fin = t;
                if (fin) {
                    // back to the start of that round (round 0: the start values, untouched)
                    for (int i = tid; i < exy * ez; i += RJ_THREADS) {
                        const int gi = global_index(i);
                        const int zz = i / exy, r = i - zz * exy, yy = r / ex;
                        const int x = lx + r - yy * ex, y = ly + yy, z = lz + zz;
                        const bool face = x == 0 || x == g.nx - 1 || y == 0 || y == g.ny - 1 || z == 0 || z == g.nz - 1;
                        if (face) continue;
                        cur[i] = past == 0 ? __ldcg(buf0 + gi) : value(look(ring + (past % RJ_RING) * g.N + gi));
                    }
                    __syncthreads();
                    double* res = past == 0 ? buf1 : buf0;
                    double md = 0.0;
                    for (int t = 1; t <= fin; ++t) {
                        const Run u = run_of(t, fin);
                        md = sweep(cur, nxt, u, nullptr, 0);
                        if (t == fin && u.n) {
                            const int gi = global_index(u.li);
                            for (int i = 0; i < u.n; ++i) res[gi + i * sxy] = nxt[u.li + i * exy];
                        }
                        __syncthreads();
                        double* q = cur;
                        cur = nxt;
                        nxt = q;
                    }
                    md = warp_max(md);
                    if (lane == 0) atomicMax(&ctrl->last_diff, (unsigned long long)__double_as_longlong(md));
                    if (b == 0 && tid == 0) {
                        ctrl->sweeps = past * T + fin;
                        ctrl->in_buf1 = past == 0;
                    }
                    return;
                }
            }
        }
        // ---- the board of round - RJ_DELAY, on its way while this round computes
        const long long seen = round - RJ_DELAY;
        const Packet* rec = board + (seen >= 0 ? seen % RJ_BOARDS : 0) * gridDim.x;
        Packet seen_of{};
        if (seen >= 0 && tid < (int)gridDim.x) seen_of = look(rec + tid);
        Packet* slot = ring + ((round + 1) % RJ_RING) * g.N + out_gi;
        unsigned over = 0;
#pragma unroll
        for (int t = 1; t <= T; ++t) {
            const double md = sweep(cur, nxt, runs[t - 1], t == T ? slot : nullptr, (unsigned)(round + 1));
            if (md >= tol) over |= 1u << (t - 1);
            if (t == T) {
                over = __reduce_or_sync(0xffffffffu, over);
                if (lane == 0 && over) atomicOr(&s_mine[round & 1], over);
            }
            __syncthreads();
            if (t == 1 && tid == 0) s_over[(round + 1) & 1] = 0;  // read by all before this sweep
            double* q = cur;
            cur = nxt;
            nxt = q;
        }
        if (tid == 0) {
            post(board + (round % RJ_BOARDS) * gridDim.x + b, __longlong_as_double((long long)s_mine[round & 1]),
                 (unsigned)(round + 1));
            s_mine[(round + 1) & 1] = 0;  // last read by this thread a round ago
        }
        if (seen >= 0 && warp * 32 < (int)gridDim.x) {
            unsigned any = 0;
            if (tid < (int)gridDim.x) {
                long long polls = 0;
                while (!has(seen_of, (unsigned)(seen + 1))) {
                    if (++polls >= poll_limit || ((polls & 1023) == 0 && atomicAdd(&ctrl->error, 0) != 0)) {
                        atomicExch(&ctrl->error, 1);
                        s_fail = 1;
                        break;
                    }
                    seen_of = look(rec + tid);
                }
                any = (unsigned)__double_as_longlong(value(seen_of));
            }
            any = __reduce_or_sync(0xffffffffu, any);
            if (lane == 0 && any) atomicOr(&s_over[round & 1], any);
        }
    }
}

// Blocks per axis for T sweeps per round: the fewest modelled cycles per sweep.  The model was fitted to
// rounds timed on B200 with T = 2, 3 and 4 on 16^3 to 60^3 (48^3, T = 3: exchange 3,000 cycles, sweeps
// 4,240, the rest 930): 800 per sweep and 0.5 per point swept (rows padded to 16), 0.7 per halo point
// and 2,000 per round.
bool pick_shape(const Grid& g, int num_sms, int T, RJShape* best, double* cost) {
    bool found = false;
    // per axis: interior points, and points of sweep T - t (t more per side than the e owned ones)
    const int nx = g.nx - 2, ny = g.ny - 2, nz = g.nz - 2;
    const auto swept_points = [](int n, int e, int t) { return std::min(n, e + 2 * t); };
    for (int bx = 1; bx <= std::min(num_sms, nx); ++bx) {
        const int ex = (nx + bx - 1) / bx, xs = (swept_points(nx, ex, T - 1) + 15) / 16;
        if (xs > RJ_ROWS) continue;
        for (int by = 1; bx * by <= num_sms && by <= ny; ++by) {
            const int ey = (ny + by - 1) / by;
            if (xs * swept_points(ny, ey, T - 1) > RJ_ROWS) continue;
            const int bz = std::min(num_sms / (bx * by), nz), ez = (nz + bz - 1) / bz;
            const long long region =
                (long long)std::min(g.nx, ex + 2 * T) * std::min(g.ny, ey + 2 * T) * std::min(g.nz, ez + 2 * T);
            const long long halo = region - (long long)ex * ey * ez;
            if (3 * region * (long long)sizeof(double) > (long long)RJ_SMEM || halo > (long long)RJ_HALO * RJ_THREADS ||
                region * 8 < halo * 4)
                continue;
            double swept = 0.0;
            for (int t = 0; t < T; ++t)
                swept += 16.0 * ((swept_points(nx, ex, t) + 15) / 16 * swept_points(ny, ey, t)) * swept_points(nz, ez, t);
            const double c = (800.0 * T + 0.5 * swept + 0.7 * (double)halo + 2000.0) / T;
            if (!found || c < *cost) {
                found = true;
                *cost = c;
                *best = {bx, by, bz, (int)region};
            }
        }
    }
    return found;
}

}  // namespace

bool hartree_resident(dft_context* ctx, const Grid& g, const double* rho, double* start, double* other, double tol,
                      long max_sweeps, JacobiResult* res, double** result) {
    RJShape sh{};
    int T = 0;
    double cost = 0.0;
    for (int t = 2; t <= RJ_TMAX; ++t) {
        RJShape s;
        double c;
        if (pick_shape(g, ctx->num_sms, t, &s, &c) && (T == 0 || c < cost)) T = t, sh = s, cost = c;
    }
    if (T == 0) return false;
    const size_t smem = sizeof(double) * 3 * (size_t)sh.points;
    const void* fn = T == 2   ? (const void*)jacobi_resident_kernel<2>
                     : T == 3 ? (const void*)jacobi_resident_kernel<3>
                              : (const void*)jacobi_resident_kernel<4>;
    DFT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RJ_SMEM));
    const int blocks = sh.bx * sh.by * sh.bz;
    // control words, boards and the exchange ring; tags start at 0
    const size_t board_packets = (size_t)RJ_BOARDS * blocks;
    const size_t bytes = 256 + sizeof(Packet) * (board_packets + (size_t)RJ_RING * g.N);
    char* ws = (char*)ws_get(ctx, WS_JACOBI_RING, bytes);
    JacobiRCtrl* ctrl = (JacobiRCtrl*)ws;
    Packet* board = (Packet*)(ws + 256);
    Packet* ring = board + board_packets;
    DFT_CUDA(cudaMemsetAsync(ws, 0, bytes, ctx->stream));
    ExactDiv dv = exact_div(2.0 * (g.ix2 + g.iy2 + g.iz2));
    Grid gg = g;
    long long cap = max_sweeps, polls = ctx->grid_barrier_poll_limit > 0 ? ctx->grid_barrier_poll_limit : (1LL << 22);
    void* args[] = {&gg, &rho, &start, &other, &ring, &board, &ctrl, &dv, &tol, &cap, &sh, &polls};
    DFT_CUDA(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(RJ_THREADS), args, smem, ctx->stream));
    count_launch(ctx);
    JacobiRCtrl* hc = (JacobiRCtrl*)pinned(ctx, (sizeof(JacobiRCtrl) + 7) / 8);
    DFT_CUDA(cudaMemcpyAsync(hc, ctrl, sizeof(JacobiRCtrl), cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    if (hc->error) fail(DFT_CUDA_ERROR, "Jacobi halo exchange timed out");
    *result = hc->in_buf1 ? other : start;
    double last;
    std::memcpy(&last, &hc->last_diff, sizeof last);
    *res = {(long)hc->sweeps, last};
    return true;
}

}  // namespace dftb
