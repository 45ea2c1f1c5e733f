// FP64 tall-skinny products of the block eigensolver on the FP64 tensor pipe:
//   gram_fp64    C = dV A^T B            (bands x bands, summed over the grid points)
//   rotate       X = beta X + alpha V Y  (bands x points)
//   ritz_residual  R = (AV) Y - (V Y) diag(theta) and |R_b|^2, without storing V Y or (AV) Y
//
// All three read band blocks band-major (points contiguous), which is the K-contiguous operand
// layout of mma.m8n8k4.f64 for the Gram product and the N-contiguous one for the rotations, so
// fragments are loaded straight from global memory: a lane's 16-byte load covers two points, and
// since the order of the summed points (Gram) or of the output columns (rotation) is free, its
// two halves feed two MMAs without any exchange.  Measured on B200 (148 SMs, 1965 MHz):
// mma.m8n8k4.f64 sustains 37.1 TFLOP/s, plain FMA 33.0, and the MMA needs a quarter of the operand
// reads of an 8 x 8 register tile; tcgen05 has no FP64 kind.
#include <algorithm>
#include <cstring>
#include <vector>

#include "ops.h"

namespace dftb {

namespace {

// D (8 x 8) += A (8 x 4, row) B (4 x 8, col).  Lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// Two neighbouring doubles: one 16-byte load where AL says that every row starts 16-byte aligned.
template <bool AL>
__device__ __forceinline__ double2 load2(const double* p) {
    if (AL) return __ldg(reinterpret_cast<const double2*>(p));
    return make_double2(__ldg(p), __ldg(p + 1));
}

// ---------------------------------------------------------------- Gram -----------------
// A block of 8 warps (WM along the rows of A, 8 / WM along the points) owns a tile of row_blocks x 8
// rows and RN x 8 columns of C and one chunk of the points.  A warp walks its share of the chunk
// 8 KU points at a time: per 8 points up to RM A fragments and RN B fragments (one 16-byte load each)
// feed 2 RM RN MMAs.  The partial tiles along the points are added in shared memory in warp order;
// the block's tile goes to partial[chunk].
//
// Small products (nel <= GM_INLINE) add the chunks' partials in the same launch (gram_finish).
constexpr int GM_THREADS = 256;
constexpr int GM_GROUP = 16;
constexpr int GM_TICKETS = 256;  // ticket words: 1 + groups
constexpr int GM_INLINE = 1024;

// The partials of nch chunks (partial[chunk], each of them `tiles` arrivals) are added in a fixed order by the
// same launch, in two levels: the last arrival of a group of GM_GROUP chunks (ticket[1 + group]) adds the
// group's partials, the last group (ticket[0]) adds the group sums and writes scale * C.  Called by
// whole thread blocks with the chunk `at` they have just written.
__device__ __forceinline__ void gram_finish(int nel, int tiles, int nch, int at, double* partial, double scale,
                                            unsigned int* ticket, double* out) {
    const int ngroups = (nch + GM_GROUP - 1) / GM_GROUP;
    const int grp = at / GM_GROUP, c0 = grp * GM_GROUP, csz = min(GM_GROUP, nch - c0);
    double* gsum = partial + (long long)nch * nel;  // [ngroups][nel]
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket + 1 + grp, 1u) == (unsigned)(csz * tiles) - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int e = threadIdx.x; e < nel; e += blockDim.x) {
        double v[GM_GROUP];
#pragma unroll
        for (int c = 0; c < GM_GROUP; ++c) v[c] = c < csz ? __ldcg(partial + (long long)(c0 + c) * nel + e) : 0.0;
        double sum = 0.0;
#pragma unroll
        for (int c = 0; c < GM_GROUP; ++c) sum += v[c];
        gsum[(long long)grp * nel + e] = sum;
    }
    if (threadIdx.x == 0) ticket[1 + grp] = 0;  // ready for the next call
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == (unsigned)ngroups - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int e = threadIdx.x; e < nel; e += blockDim.x) {
        double sum = 0.0;
        for (int q0 = 0; q0 < ngroups; q0 += 16) {
            double v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = q0 + q < ngroups ? __ldcg(gsum + (long long)(q0 + q) * nel + e) : 0.0;
#pragma unroll
            for (int q = 0; q < 16; ++q) sum += v[q];
        }
        out[e] = sum * scale;
    }
    if (threadIdx.x == 0) *ticket = 0;
}

template <int RM, int RN>
constexpr int gram_ku() { return RM + RN <= 3 ? 4 : RM + RN <= 6 ? 2 : 1; }
template <int RM, int RN>
constexpr int gram_blocks() { return RM * RN > 18 ? 1 : 2; }  // resident blocks per SM (registers)

template <int RM, int RN, bool AL>
__global__ void __launch_bounds__(GM_THREADS, (gram_blocks<RM, RN>()))
    gram_mma_kernel(const double* __restrict__ A, long long lda, int ka, const double* __restrict__ B, long long ldb,
                    int kb, long long n, long long chunk, int wm_count, int row_blocks, double scale,
                    double* __restrict__ partial, unsigned int* __restrict__ ticket, double* __restrict__ out) {
    extern __shared__ double tile[];  // (8 row_blocks) x (8 RN + 2)
    constexpr int TS = 8 * RN + 2, KU = gram_ku<RM, RN>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp % wm_count, wk = warp / wm_count, wk_count = 8 / wm_count;
    const int g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.x * 8 * row_blocks, n0 = blockIdx.y * 8 * RN;
    const int rb = min(row_blocks, (ka - m0 + 7) / 8);  // row blocks of this tile
    // this warp's row blocks: [r0, r0 + nr), the remainder to the first warps
    const int nr = rb / wm_count + (wm < rb % wm_count);
    const int r0 = wm * (rb / wm_count) + min(wm, rb % wm_count);
    const long long p0 = (long long)blockIdx.z * chunk, p1 = min(n, p0 + chunk);
    // fragment row 8 r is read while 8 r < va (A) or vb (B); rows past the end count as zero
    const int va = min(8 * nr, ka - (m0 + 8 * r0 + g)), vb = kb - (n0 + g);
    const double* pa = A + (long long)(m0 + 8 * r0 + g) * lda;
    const double* pb = B + (long long)(n0 + g) * ldb;
    const long long a8 = 8 * lda, b8 = 8 * ldb;
    const double2 zero2 = make_double2(0.0, 0.0);
    double acc[RM][RN][2];
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[r][j][0] = acc[r][j][1] = 0.0;
    const long long step = 8LL * KU * wk_count;
    const long long full = p0 + (p1 - p0) / (8 * KU) * (8 * KU);  // end of the whole slices
    long long p = p0 + 8LL * KU * wk;
    if (nr > 0)
        for (; p < full; p += step) {
            double2 a[KU][RM], b[KU][RN];
#pragma unroll
            for (int u = 0; u < KU; ++u) {
#pragma unroll
                for (int r = 0; r < RM; ++r)
                    a[u][r] = 8 * r < va ? load2<AL>(pa + r * a8 + p + 8 * u + 2 * t) : zero2;
#pragma unroll
                for (int j = 0; j < RN; ++j)
                    b[u][j] = 8 * j < vb ? load2<AL>(pb + j * b8 + p + 8 * u + 2 * t) : zero2;
            }
#pragma unroll
            for (int u = 0; u < KU; ++u)
#pragma unroll
                for (int r = 0; r < RM; ++r) {
                    if (r >= nr) break;
#pragma unroll
                    for (int j = 0; j < RN; ++j) mma_f64(acc[r][j], a[u][r].x, b[u][j].x);
#pragma unroll
                    for (int j = 0; j < RN; ++j) mma_f64(acc[r][j], a[u][r].y, b[u][j].y);
                }
        }
    if (nr > 0 && p == full)  // the warp whose turn it is takes the ragged end, four points at a time
        for (; p < p1; p += 4) {
            const bool in = p + t < p1;
            double a[RM], b[RN];
#pragma unroll
            for (int r = 0; r < RM; ++r) a[r] = in && 8 * r < va ? __ldg(pa + r * a8 + p + t) : 0.0;
#pragma unroll
            for (int j = 0; j < RN; ++j) b[j] = in && 8 * j < vb ? __ldg(pb + j * b8 + p + t) : 0.0;
#pragma unroll
            for (int r = 0; r < RM; ++r)
#pragma unroll
                for (int j = 0; j < RN; ++j) mma_f64(acc[r][j], a[r], b[j]);
        }
    for (int w = 0; w < wk_count; ++w) {
        if (wk == w)
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                if (r >= nr) break;
#pragma unroll
                for (int j = 0; j < RN; ++j) {
                    double* c = tile + ((r0 + r) * 8 + g) * TS + j * 8 + 2 * t;
                    c[0] = w ? c[0] + acc[r][j][0] : acc[r][j][0];
                    c[1] = w ? c[1] + acc[r][j][1] : acc[r][j][1];
                }
            }
        __syncthreads();
    }
    const int nel = ka * kb;
    double* mine = partial + (long long)blockIdx.z * nel;
    const int rows = min(8 * row_blocks, ka - m0), cols = min(8 * RN, kb - n0);
    for (int e = threadIdx.x; e < rows * cols; e += GM_THREADS) {
        const int i = e / cols, j = e - i * cols;
        mine[(long long)(m0 + i) * kb + n0 + j] = tile[i * TS + j];
    }
    if (ticket)
        gram_finish(nel, (int)(gridDim.x * gridDim.y), (int)gridDim.z, (int)blockIdx.z, partial, scale, ticket, out);
}

// out[e] = scale * sum_c partial[c][e] for wide products: 32 neighbouring elements by 8 strands of
// chunks per block (coalesced), the strands added in order.
__global__ void __launch_bounds__(256) gram_sum_kernel(int nch, int nel, const double* __restrict__ partial,
                                                       double scale, double* __restrict__ out) {
    __shared__ double sh[8][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + x;
    double s = 0.0;
    if (e < nel)
#pragma unroll 4
        for (int c = y; c < nch; c += 8) s += partial[(long long)c * nel + e];
    sh[y][x] = s;
    __syncthreads();
    if (y == 0 && e < nel) {
        s = sh[0][x];
#pragma unroll
        for (int q = 1; q < 8; ++q) s += sh[q][x];
        out[e] = s * scale;
    }
}

// ---------------------------------------------------------------- ordered Gram ---------
// Blocks of up to 64 x 16 (the eigensolver of a small molecule) keep a fixed order of summation, so that
// nothing downstream that turns on the last bit (the sign of an eigenvector of the projected
// matrix) depends on how the work is split.  On this chip an MMA adds its four products one after the
// other like four FMAs (nothing promises it; the tests hold these products to the chains bit for
// bit), so a chain of MMAs along the points is the scalar chain; each element is a set of such chains,
// added in a fixed tree.
//
// gram_lanes_kernel (kb <= 4, 8 or 16 with ka <= 64, 64, 32): the points are dealt to nblk blocks of 32
// chains; chain (b, l) takes the points 32 b + l + 32 m nblk.  The 32 chains of block b are added as a
// butterfly (xor 16, 8, 4, 2, 1), then the blocks in order, GM_GROUP at a time.  A thread block works
// through its blocks b in turn; 4 U m of 32 points and all rows are staged ahead in shared memory by
// cp.async (reading fragments straight from global memory costs 32 L1 lookups per load, one per
// row and m: 50 us for 24 x 12 at 64^3).  A warp runs two chains for all RB x CB tiles.  The 272-byte pitch of
// a staged 256-byte segment makes the 16-byte fragment reads free of bank conflicts.
// 64^3, 24 x 12: 93 us with one FMA per lane and product, 36 us here.
constexpr int GL_PITCH = 272;  // bytes per staged segment (row, m)

__device__ __forceinline__ void stage(void* dst, const void* src, bool wide, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int RB, int CB>
struct LanesShape {
    static constexpr int ROWS = 8 * (RB + CB), SUM = 16 * RB * CB * 64 * 8;
    // groups of four m per stage: few rows make short stages, whose barriers then take the time (128^3, one group / as
    // here: 2 x 2 82 / 52 us, 8 x 8 95 / 72)
    static constexpr int U = ROWS <= 16 ? 4 : ROWS <= 24 ? 2 : 1;
    static constexpr int PITCH = 4 * U * GL_PITCH + (U > 1 ? 64 : 0);  // of a row: 16 banks apart
    static constexpr int STAGE = ROWS * PITCH;
    static constexpr int S = (220 * 1024 - SUM) / STAGE >= 4 ? 4 : (220 * 1024 - SUM) / STAGE;  // stages in flight
    static constexpr size_t SMEM = (size_t)S * STAGE + SUM;
};

template <int RB, int CB, bool AL>
__global__ void __launch_bounds__(512, 1)
    gram_lanes_kernel(const double* __restrict__ A, long long lda, int ka, const double* __restrict__ B, long long ldb,
                      int kb, long long n, int nblk, double* __restrict__ partial) {
    using Shape = LanesShape<RB, CB>;
    extern __shared__ __align__(16) char stages[];  // S x (8 (RB + CB) rows) x 4 U m; then the butterfly's sums
    constexpr int TILES = RB * CB, STAGE = Shape::STAGE, S = Shape::S, U = Shape::U, M = 4 * U;
    double* sum = reinterpret_cast<double*>(stages + S * STAGE);  // 8 warps x 2 chains x TILES x 64
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long stride = (long long)nblk * 32;
    const int steps = (int)((n + M * stride - 1) / (M * stride));  // per block b (the last ones may be empty)
    const int nb = ((int)blockIdx.x < nblk) ? (nblk - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = nb * steps;
    // stage q of this thread block: step q % steps of its block number q / steps
    auto fill = [&](int q) {
        if (q < total) {
            const int b = (int)blockIdx.x + q / steps * (int)gridDim.x, s = q % steps;
            char* to = stages + q % S * STAGE;
            constexpr int PER = AL ? 16 : 32;  // copies per segment
            // (rows that do not exist are not staged: what their shared memory holds reaches only elements that
            // are not stored; 20 x 4 at 128^3 with zeros in their place 183 us, 131 here)
            for (int e = threadIdx.x; e < (ka + kb) * M * PER; e += 512) {
                const int c = e % PER, m = e / PER % M, r = e / (M * PER);
                const bool of_a = r < ka;
                const double* base = of_a ? A + (long long)r * lda : B + (long long)(r - ka) * ldb;
                const int row = of_a ? r : 8 * RB + r - ka;
                const long long p = (long long)b * 32 + (long long)(M * s + m) * stride + c * (AL ? 2 : 1);
                const int in = p >= n ? 0 : AL ? (p + 1 < n ? 16 : 8) : 8;
                stage(to + row * Shape::PITCH + m * GL_PITCH + c * (AL ? 16 : 8), in ? base + p : base, AL, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[2][TILES][2];
    for (int q = 0; q < S - 1; ++q) fill(q);
    for (int q = 0; q < total; ++q) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncthreads();  // stage q has landed, and everyone is done with stage q - 1
        fill(q + S - 1);
        if (q % steps == 0)
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int x = 0; x < TILES; ++x) acc[c][x][0] = acc[c][x][1] = 0.0;
        const char* from = stages + q % S * STAGE + t * GL_PITCH + warp * 16;
#pragma unroll
        for (int u = 0; u < U; ++u, from += 4 * GL_PITCH) {
            double2 a[RB], b[CB];
#pragma unroll
            for (int r = 0; r < RB; ++r) a[r] = *reinterpret_cast<const double2*>(from + (8 * r + g) * Shape::PITCH);
#pragma unroll
            for (int j = 0; j < CB; ++j) b[j] = *reinterpret_cast<const double2*>(from + (8 * (RB + j) + g) * Shape::PITCH);
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    mma_f64(acc[0][r * CB + j], a[r].x, b[j].x);
                    mma_f64(acc[1][r * CB + j], a[r].y, b[j].y);
                }
        }
        if (q % steps != steps - 1) continue;
        // butterfly over the block's 32 chains: chain 2 w + c is in warp w
#pragma unroll
        for (int half = 8; half >= 1; half >>= 1) {
            if (warp >= half && warp < 2 * half) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int x = 0; x < TILES; ++x)
                        reinterpret_cast<double2*>(sum)[(((warp - half) * 2 + c) * TILES + x) * 32 + lane] =
                            make_double2(acc[c][x][0], acc[c][x][1]);
            }
            __syncthreads();
            if (warp < half) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int x = 0; x < TILES; ++x) {
                        const double2 o = reinterpret_cast<double2*>(sum)[((warp * 2 + c) * TILES + x) * 32 + lane];
                        acc[c][x][0] += o.x;
                        acc[c][x][1] += o.y;
                    }
            }
            __syncthreads();
        }
        const int nel = ka * kb, blk = (int)blockIdx.x + q / steps * (int)gridDim.x;
        if (warp == 0) {
            double* mine = partial + (long long)blk * nel;
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int j = 0; j < CB; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = 8 * r + g, k = 8 * j + 2 * t + h;
                        if (i < ka && k < kb) mine[i * kb + k] = acc[0][r * CB + j][h] + acc[1][r * CB + j][h];
                    }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// out[e] = scale * the blocks' partials, added GM_GROUP blocks at a time in block order, then the groups in order
constexpr int GL_GROUPS = 64;  // at most 64 x 16 blocks
__global__ void __launch_bounds__(8 * GL_GROUPS) gram_lanes_sum_kernel(int nblk, int nel,
                                                                       const double* __restrict__ partial, double scale,
                                                                       double* __restrict__ out) {
    __shared__ double sh[GL_GROUPS][8];
    const int e = blockIdx.x * 8 + threadIdx.x, grp = threadIdx.y, groups = blockDim.y;
    if (e < nel) {
        double v[GM_GROUP];
#pragma unroll
        for (int c = 0; c < GM_GROUP; ++c)
            v[c] = grp * GM_GROUP + c < nblk ? __ldg(partial + (long long)(grp * GM_GROUP + c) * nel + e) : 0.0;
        double sum = 0.0;
#pragma unroll
        for (int c = 0; c < GM_GROUP; ++c) sum += v[c];
        sh[grp][threadIdx.x] = sum;
    }
    __syncthreads();
    if (grp || e >= nel) return;
    double sum = 0.0;
    for (int q = 0; q < groups; ++q) sum += sh[q][threadIdx.x];
    out[e] = sum * scale;
}

// gram_chunk_kernel (the other blocks up to 64 x 16): one chain per chunk of the points and element.  Warp w
// owns row tile w; a chunk's points in order, 4 per MMA, eight steps of loads in flight.
template <int CB>
__global__ void __launch_bounds__(256, 2)
    gram_chunk_kernel(const double* __restrict__ A, long long lda, int ka, const double* __restrict__ B, long long ldb,
                      int kb, long long n, long long chunk, double* __restrict__ partial) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long p0 = (long long)blockIdx.x * chunk, p1 = min(n, p0 + chunk);
    const int i = 8 * warp + g, vb = kb - g;
    const double* pa = A + (long long)(i < ka ? i : 0) * lda;
    const double* pb = B + (long long)g * ldb;
    double acc[CB][2];
#pragma unroll
    for (int j = 0; j < CB; ++j) acc[j][0] = acc[j][1] = 0.0;
    constexpr int U = 8;
    for (long long p = p0; p < p1; p += 4 * U) {
        double a[U], b[U][CB];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long q = p + 4 * u + t;
            a[u] = q < p1 && i < ka ? __ldg(pa + q) : 0.0;
#pragma unroll
            for (int j = 0; j < CB; ++j) b[u][j] = q < p1 && 8 * j < vb ? __ldg(pb + 8 * j * ldb + q) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < CB; ++j) mma_f64(acc[j], a[u], b[u][j]);
    }
    double* mine = partial + (long long)blockIdx.x * ka * kb;
#pragma unroll
    for (int j = 0; j < CB; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 8 * j + 2 * t + h;
            if (i < ka && k < kb) mine[i * kb + k] = acc[j][h];
        }
}

// out[e] = scale * sum_c partial[c][e]: one warp per element, lanes stride the chunks, butterfly
__global__ void __launch_bounds__(256) gram_chunk_sum_kernel(int nch, int nel, const double* __restrict__ partial,
                                                             double scale, double* __restrict__ out) {
    const int lane = threadIdx.x & 31, e = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (e >= nel) return;
    double s = 0.0;
#pragma unroll 4
    for (int c = lane; c < nch; c += 32) s += partial[(long long)c * nel + e];
    s = warp_sum(s);
    if (lane == 0) out[e] = s * scale;
}

unsigned int* gram_tickets(dft_context* ctx) {
    if (!ctx->gram_ticket) {
        DFT_CUDA(cudaMalloc(&ctx->gram_ticket, sizeof(unsigned int) * GM_TICKETS));
        DFT_CUDA(cudaMemsetAsync(ctx->gram_ticket, 0, sizeof(unsigned int) * GM_TICKETS, ctx->stream));
    }
    return (unsigned int*)ctx->gram_ticket;
}

void gram_to_host(dft_context* ctx, const double* res, size_t nel, std::vector<double>& C) {
    double* h = pinned(ctx, nel);
    DFT_CUDA(cudaMemcpyAsync(h, res, sizeof(double) * nel, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    std::memcpy(C.data(), h, sizeof(double) * nel);
}

template <int RB, int CB, bool AL>
void gram_lanes(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B, long long ldb,
                int kb, std::vector<double>& C) {
    const size_t nel = (size_t)ka * kb;
    const int nblk = (int)std::max<long long>(
        1, std::min<long long>(std::min(4LL * ctx->num_sms, (long long)GL_GROUPS * GM_GROUP), (g.N + 255) / 256));
    const int ngroups = (nblk + GM_GROUP - 1) / GM_GROUP;
    double* partial = (double*)ws_get(ctx, WS_SMALL, sizeof(double) * (nel * nblk + nel));
    double* res = partial + nel * nblk;
    constexpr size_t smem = LanesShape<RB, CB>::SMEM;
    DFT_CUDA(cudaFuncSetAttribute(gram_lanes_kernel<RB, CB, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    gram_lanes_kernel<RB, CB, AL><<<std::min(nblk, ctx->num_sms), 512, smem, ctx->stream>>>(
        A, lda, ka, B, ldb, kb, g.N, nblk, partial);
    DFT_LAUNCH_CHECK();
    gram_lanes_sum_kernel<<<(unsigned)((nel + 7) / 8), dim3(8, ngroups), 0, ctx->stream>>>(nblk, (int)nel, partial, g.dV,
                                                                                            res);
    DFT_LAUNCH_CHECK();
    count_launch(ctx, 2);
    gram_to_host(ctx, res, nel, C);
}

// ka <= 64 and kb <= 16
template <bool AL>
void gram_ordered(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B,
                  long long ldb, int kb, std::vector<double>& C) {
    // the row counts and column widths at which the order changes
    const int rows = ka <= 8 ? 1 : ka <= 16 ? 2 : ka <= 32 ? 4 : 8, cols = kb <= 4 ? 4 : kb <= 8 ? 8 : 16;
    if (rows * cols <= 64) {
        switch (rows * 10 + (cols + 7) / 8) {
            case 11: gram_lanes<1, 1, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            case 12: gram_lanes<1, 2, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            case 21: gram_lanes<2, 1, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            case 22: gram_lanes<2, 2, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            case 41: gram_lanes<4, 1, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            case 42: gram_lanes<4, 2, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
            default: gram_lanes<8, 1, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); return;
        }
    }
    const size_t nel = (size_t)ka * kb;
    const int tiles = (ka + 31) / 32;
    long long nch = std::max<long long>(1, 4LL * ctx->num_sms / tiles);
    long long chunk = ((g.N + nch - 1) / nch + 31) / 32 * 32;
    nch = std::min<long long>((g.N + chunk - 1) / chunk, 65535);
    chunk = (g.N + nch - 1) / nch;
    double* partial = (double*)ws_get(ctx, WS_SMALL, sizeof(double) * (nel * nch + nel));
    double* res = partial + nel * nch;
    const int threads = 32 * ((ka + 7) / 8);
    if (kb <= 8)
        gram_chunk_kernel<1><<<(unsigned)nch, threads, 0, ctx->stream>>>(A, lda, ka, B, ldb, kb, g.N, chunk, partial);
    else
        gram_chunk_kernel<2><<<(unsigned)nch, threads, 0, ctx->stream>>>(A, lda, ka, B, ldb, kb, g.N, chunk, partial);
    DFT_LAUNCH_CHECK();
    gram_chunk_sum_kernel<<<(unsigned)((nel + 7) / 8), 256, 0, ctx->stream>>>((int)nch, (int)nel, partial, g.dV, res);
    DFT_LAUNCH_CHECK();
    count_launch(ctx, 2);
    gram_to_host(ctx, res, nel, C);
}

template <int RM, int RN, bool AL>
void gram_launch(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B,
                 long long ldb, int kb, std::vector<double>& C) {
    constexpr int KU = gram_ku<RM, RN>();
    // row tiles of at most 8 warps x RM blocks of 8 rows, all of one height; the fewest warps along M
    // that hold a tile (the others split the points)
    const int blocks = (ka + 7) / 8, mt = (blocks + 8 * RM - 1) / (8 * RM);
    const int row_blocks = (blocks + mt - 1) / mt;
    int wm = 1;
    while (wm * RM < row_blocks) wm *= 2;
    const int nt = (kb + 8 * RN - 1) / (8 * RN);
    const size_t smem = sizeof(double) * 8 * row_blocks * (8 * RN + 2);
    // one wave of blocks: as many point chunks as fit the resident blocks, none shorter than two
    // steps of every warp
    const long long resident = (long long)gram_blocks<RM, RN>() * ctx->num_sms;
    const long long unit = 8LL * KU * (8 / wm);
    long long nch = std::max<long long>(1, resident / ((long long)mt * nt));
    nch = std::min(nch, std::max<long long>(1, g.N / (2 * unit)));
    const size_t nel = (size_t)ka * kb;
    const bool inl = nel <= GM_INLINE;
    if (inl) nch = std::min<long long>(nch, (long long)(GM_TICKETS - 1) * GM_GROUP);
    nch = std::min<long long>(nch, 65535);
    long long chunk = (g.N + nch - 1) / nch;
    chunk = (chunk + unit - 1) / unit * unit;
    nch = (g.N + chunk - 1) / chunk;
    const long long ngroups = inl ? (nch + GM_GROUP - 1) / GM_GROUP : 0;
    double* partial = (double*)ws_get(ctx, WS_SMALL, sizeof(double) * (nel * (nch + ngroups) + nel) + 64);
    double* res = partial + nel * (nch + ngroups);
    if (smem > 48 * 1024)
        DFT_CUDA(cudaFuncSetAttribute(gram_mma_kernel<RM, RN, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(sizeof(double) * 64 * RM * (8 * RN + 2))));
    gram_mma_kernel<RM, RN, AL><<<dim3(mt, nt, (unsigned)nch), GM_THREADS, smem, ctx->stream>>>(
        A, lda, ka, B, ldb, kb, g.N, chunk, wm, row_blocks, g.dV, partial,
        inl ? gram_tickets(ctx) : nullptr, res);
    DFT_LAUNCH_CHECK();
    if (!inl) {
        gram_sum_kernel<<<(unsigned)((nel + 31) / 32), 256, 0, ctx->stream>>>((int)nch, (int)nel, partial, g.dV, res);
        DFT_LAUNCH_CHECK();
    }
    count_launch(ctx, inl ? 1 : 2);
    gram_to_host(ctx, res, nel, C);
}

template <int RN, bool AL>
void gram_rows(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B, long long ldb,
               int kb, std::vector<double>& C) {
    // blocks of 8 rows per warp: as few as one warp column can hold up to 4, which shares each B
    // fragment best
    if (ka <= 8) gram_launch<1, RN, AL>(ctx, g, A, lda, ka, B, ldb, kb, C);
    else if (ka <= 16) gram_launch<2, RN, AL>(ctx, g, A, lda, ka, B, ldb, kb, C);
    else gram_launch<4, RN, AL>(ctx, g, A, lda, ka, B, ldb, kb, C);
}

template <bool AL>
void gram_pick(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B, long long ldb,
               int kb, std::vector<double>& C) {
    if (ka <= 64 && kb <= 16) {
        gram_ordered<AL>(ctx, g, A, lda, ka, B, ldb, kb, C);
        return;
    }
    // columns: tiles of at most 72, all of the same width
    const int tiles = (kb + 71) / 72;
    switch ((((kb + tiles - 1) / tiles) + 7) / 8) {
        case 1: gram_rows<1, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 2: gram_rows<2, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 3: gram_rows<3, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 4: gram_rows<4, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 5: gram_rows<5, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 6: gram_rows<6, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 7: gram_rows<7, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        case 8: gram_rows<8, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
        default: gram_rows<9, AL>(ctx, g, A, lda, ka, B, ldb, kb, C); break;
    }
}

// every row of the block starts 16-byte aligned
inline bool aligned16(const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 2 == 0; }

}  // namespace

// C (ka x kb, host, row-major) = dV * A^T B
void gram_fp64(dft_context* ctx, const Grid& g, const double* A, long long lda, int ka, const double* B, long long ldb,
               int kb, std::vector<double>& C) {
    C.assign((size_t)ka * kb, 0.0);
    if (ka == 0 || kb == 0) return;
    if (aligned16(A, lda) && aligned16(B, ldb)) gram_pick<true>(ctx, g, A, lda, ka, B, ldb, kb, C);
    else gram_pick<false>(ctx, g, A, lda, ka, B, ldb, kb, C);
}

namespace {

// ---------------------------------------------------------------- rotation -------------
// out_j = beta out_j + alpha sum_i in_i Y[i][j] over i < k, for 8 RJ columns j from j0 = 8 RJ blockIdx.y.
// A warp owns 16 PP points and all 8 RJ columns, so `in` is read once; per 4 rows of `in` it loads
// PP 16-byte pairs of points per lane and RJ fragments of Y^T from shared memory for 2 PP RJ MMAs.
// Y^T is laid out in fragment order (conflict-free).  The two points of a pair go to two MMAs, so
// a lane ends with four neighbouring points of one column.
// in2: the rows k1 <= i < k come from in2 (row i - k1).  ss: when not null, sum_p out_j[p]^2 of
// this block goes to ss[j * gridDim.x + blockIdx.x].
// out may be rows of `in` when one column tile covers all of m (rotate_in_place): a warp has read
// every row at its points before it writes any of them, and no other warp reads those points.
template <int RJ, int PP, bool AL>
__global__ void __launch_bounds__(512, 1)
    rotate_mma_kernel(const double* in, const double* in2, long long ldi, int k1, int k,
                      const double* __restrict__ Y, int m, double* out, long long ldo, long long n,
                      double alpha, double beta, double* __restrict__ ss) {
    extern __shared__ double sy[];  // ceil(k / 4) x RJ x 32
    __shared__ double red[16][8 * RJ];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int j0 = blockIdx.y * 8 * RJ;
    const int steps = (k + 3) / 4;
    for (int e = threadIdx.x; e < steps * RJ * 32; e += blockDim.x) {
        const int l = e & 31, b = (e >> 5) % RJ, s = (e >> 5) / RJ;
        const int i = 4 * s + (l & 3), j = j0 + 8 * b + (l >> 2);
        sy[e] = i < k && j < m ? Y[(long long)i * m + j] : 0.0;
    }
    __syncthreads();
    double sq[RJ];
#pragma unroll
    for (int b = 0; b < RJ; ++b) sq[b] = 0.0;
    const double2 zero2 = make_double2(0.0, 0.0);
    const long long tiles = (n + 16 * PP - 1) / (16 * PP);
    for (long long tile = (long long)blockIdx.x * warps + warp; tile < tiles; tile += (long long)gridDim.x * warps) {
        const long long p0 = tile * 16 * PP;
        const bool whole = p0 + 16 * PP <= n;
        double acc[RJ][PP][2][2];
#pragma unroll
        for (int b = 0; b < RJ; ++b)
#pragma unroll
            for (int q = 0; q < PP; ++q) acc[b][q][0][0] = acc[b][q][0][1] = acc[b][q][1][0] = acc[b][q][1][1] = 0.0;
        auto fetch = [&](int s, double2 (&v)[PP]) {
            const int i = 4 * s + t;
            const double* row = (i < k1 ? in + (long long)i * ldi : in2 + (long long)(i - k1) * ldi) + p0 + 2 * g;
#pragma unroll
            for (int q = 0; q < PP; ++q) {
                if (i >= k) {
                    v[q] = zero2;
                } else if (whole) {
                    v[q] = AL ? *reinterpret_cast<const double2*>(row + 16 * q)
                              : make_double2(row[16 * q], row[16 * q + 1]);
                } else {
                    const long long p = p0 + 16 * q + 2 * g;
                    v[q].x = p < n ? row[16 * q] : 0.0;
                    v[q].y = p + 1 < n ? row[16 * q + 1] : 0.0;
                }
            }
        };
        auto product = [&](int s, const double2 (&v)[PP]) {
            const double* a = sy + (s * RJ) * 32 + lane;
#pragma unroll
            for (int b = 0; b < RJ; ++b) {
                const double y = a[b * 32];
#pragma unroll
                for (int q = 0; q < PP; ++q) {
                    mma_f64(acc[b][q][0], y, v[q].x);
                    mma_f64(acc[b][q][1], y, v[q].y);
                }
            }
        };
        // four steps (16 rows of `in`) in flight
        int s = 0;
        for (; s + 4 <= steps; s += 4) {
            double2 v[4][PP];
#pragma unroll
            for (int u = 0; u < 4; ++u) fetch(s + u, v[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u) product(s + u, v[u]);
        }
        for (; s < steps; ++s) {
            double2 v[PP];
            fetch(s, v);
            product(s, v);
        }
#pragma unroll
        for (int b = 0; b < RJ; ++b) {
            const int j = j0 + 8 * b + g;
            if (j >= m) continue;
#pragma unroll
            for (int q = 0; q < PP; ++q) {
                const long long p = p0 + 16 * q + 4 * t;
                double* o = out + (long long)j * ldo + p;
                double r[4] = {acc[b][q][0][0], acc[b][q][1][0], acc[b][q][0][1], acc[b][q][1][1]};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    r[c] *= alpha;
                    if (beta != 0.0 && p + c < n) r[c] += beta * o[c];
                    if (p + c < n) sq[b] += r[c] * r[c];
                }
                if (AL && whole) {
                    reinterpret_cast<double2*>(o)[0] = make_double2(r[0], r[1]);
                    reinterpret_cast<double2*>(o)[1] = make_double2(r[2], r[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (p + c < n) o[c] = r[c];
                }
            }
        }
    }
    if (!ss) return;
#pragma unroll
    for (int b = 0; b < RJ; ++b) {
        sq[b] += __shfl_xor_sync(0xffffffffu, sq[b], 1);
        sq[b] += __shfl_xor_sync(0xffffffffu, sq[b], 2);
        if (t == 0) red[warp][8 * b + g] = sq[b];
    }
    __syncthreads();
    if (threadIdx.x < 8 * RJ && j0 + (int)threadIdx.x < m) {
        double v = red[0][threadIdx.x];
        for (int w = 1; w < warps; ++w) v += red[w][threadIdx.x];
        ss[(long long)(j0 + threadIdx.x) * gridDim.x + blockIdx.x] = v;
    }
}

// R_b = sum_i AV_i Y[i][b] - theta_b sum_i V_i Y[i][b], the two sums kept apart and rounded once each as
// if (AV) Y and V Y had been formed; layout and ss as in rotate_mma_kernel.
template <int RJ, int PP, bool AL>
__global__ void __launch_bounds__(512, 1)
    residual_mma_kernel(const double* __restrict__ AV, const double* __restrict__ V, long long ld, int k,
                        const double* __restrict__ Y, const double* __restrict__ theta, int m, double* __restrict__ R,
                        long long n, double* __restrict__ ss) {
    extern __shared__ double sy[];  // ceil(k / 4) x RJ x 32
    __shared__ double red[16][8 * RJ];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int steps = (k + 3) / 4;
    for (int e = threadIdx.x; e < steps * RJ * 32; e += blockDim.x) {
        const int l = e & 31, b = (e >> 5) % RJ, s = (e >> 5) / RJ;
        const int i = 4 * s + (l & 3), j = 8 * b + (l >> 2);
        sy[e] = i < k && j < m ? Y[(long long)i * m + j] : 0.0;
    }
    __syncthreads();
    double sq[RJ], th[RJ];
#pragma unroll
    for (int b = 0; b < RJ; ++b) {
        sq[b] = 0.0;
        th[b] = 8 * b + g < m ? theta[8 * b + g] : 0.0;
    }
    const long long tiles = (n + 16 * PP - 1) / (16 * PP);
    for (long long tile = (long long)blockIdx.x * warps + warp; tile < tiles; tile += (long long)gridDim.x * warps) {
        const long long p0 = tile * 16 * PP;
        const bool whole = p0 + 16 * PP <= n;
        double acc[2][RJ][PP][2][2];  // AV, V
#pragma unroll
        for (int f = 0; f < 2; ++f)
#pragma unroll
            for (int b = 0; b < RJ; ++b)
#pragma unroll
                for (int q = 0; q < PP; ++q)
                    acc[f][b][q][0][0] = acc[f][b][q][0][1] = acc[f][b][q][1][0] = acc[f][b][q][1][1] = 0.0;
        auto fetch = [&](const double* F, int s, double2 (&v)[PP]) {
            const int i = 4 * s + t;
            const double* row = F + (long long)i * ld + p0 + 2 * g;
#pragma unroll
            for (int q = 0; q < PP; ++q) {
                if (i >= k) {
                    v[q] = make_double2(0.0, 0.0);
                } else if (whole) {
                    v[q] = load2<AL>(row + 16 * q);
                } else {
                    const long long p = p0 + 16 * q + 2 * g;
                    v[q].x = p < n ? __ldg(row + 16 * q) : 0.0;
                    v[q].y = p + 1 < n ? __ldg(row + 16 * q + 1) : 0.0;
                }
            }
        };
        constexpr int U = 2;
        for (int s = 0; s < steps; s += U) {
            double2 v[U][2][PP];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                fetch(AV, s + u, v[u][0]);
                fetch(V, s + u, v[u][1]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (s + u >= steps) break;
                const double* a = sy + ((s + u) * RJ) * 32 + lane;
#pragma unroll
                for (int b = 0; b < RJ; ++b) {
                    const double y = a[b * 32];
#pragma unroll
                    for (int f = 0; f < 2; ++f)
#pragma unroll
                        for (int q = 0; q < PP; ++q) {
                            mma_f64(acc[f][b][q][0], y, v[u][f][q].x);
                            mma_f64(acc[f][b][q][1], y, v[u][f][q].y);
                        }
                }
            }
        }
#pragma unroll
        for (int b = 0; b < RJ; ++b) {
            const int j = 8 * b + g;
            if (j >= m) continue;
#pragma unroll
            for (int q = 0; q < PP; ++q) {
                const long long p = p0 + 16 * q + 4 * t;
                double* o = R + (long long)j * ld + p;
                double r[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    r[c] = fma(-th[b], acc[1][b][q][c & 1][c >> 1], acc[0][b][q][c & 1][c >> 1]);
                    if (p + c < n) sq[b] += r[c] * r[c];
                }
                if (AL && whole) {
                    reinterpret_cast<double2*>(o)[0] = make_double2(r[0], r[1]);
                    reinterpret_cast<double2*>(o)[1] = make_double2(r[2], r[3]);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (p + c < n) o[c] = r[c];
                }
            }
        }
    }
#pragma unroll
    for (int b = 0; b < RJ; ++b) {
        sq[b] += __shfl_xor_sync(0xffffffffu, sq[b], 1);
        sq[b] += __shfl_xor_sync(0xffffffffu, sq[b], 2);
        if (t == 0) red[warp][8 * b + g] = sq[b];
    }
    __syncthreads();
    if ((int)threadIdx.x < min(8 * RJ, m)) {
        double v = red[0][threadIdx.x];
        for (int w = 1; w < warps; ++w) v += red[w][threadIdx.x];
        ss[(long long)threadIdx.x * gridDim.x + blockIdx.x] = v;
    }
}

// out[r] = sum of row r of partial (one block per row, fixed order)
__global__ void __launch_bounds__(128) row_sum_kernel(int ncols, const double* __restrict__ partial,
                                                      double* __restrict__ out) {
    __shared__ double sh[4];
    double s = 0.0;
    for (int c = threadIdx.x; c < ncols; c += 128) s += partial[(long long)blockIdx.x * ncols + c];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

constexpr size_t ROT_SMEM = 200 * 1024;

template <int RJ, int PP, bool AL>
unsigned rotate_launch(dft_context* ctx, const double* in, const double* in2, long long ldi, int k1, int k,
                       const double* Y, int m, double* out, long long ldo, long long n, double alpha, double beta,
                       double* ss) {
    const size_t smem = sizeof(double) * (size_t)((k + 3) / 4) * RJ * 32;
    if (smem > 32 * 1024) {  // with the 9 KB of static shared memory beyond the default limit
        DFT_CUDA(cudaFuncSetAttribute(rotate_mma_kernel<RJ, PP, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)ROT_SMEM));
    }
    const int jt = (m + 8 * RJ - 1) / (8 * RJ);
    // 16 warps per SM (the register limit): as two blocks, or as one where Y^T takes most of the
    // shared memory
    const int threads = smem > 90 * 1024 ? 512 : 256;
    const long long warps_needed = (n + 16 * PP - 1) / (16 * PP);
    const long long resident = (long long)ctx->num_sms * 512 / threads;
    const long long bx = std::max<long long>(
        1, std::min<long long>((warps_needed * 32 + threads - 1) / threads, (resident + jt - 1) / jt));
    rotate_mma_kernel<RJ, PP, AL><<<dim3((unsigned)bx, jt), threads, smem, ctx->stream>>>(in, in2, ldi, k1, k, Y, m,
                                                                                         out, ldo, n, alpha, beta, ss);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    return (unsigned)bx;
}

// most blocks along x that rotate_launch uses (the row length of ss)
inline size_t rotate_max_blocks(dft_context* ctx) { return (size_t)ctx->num_sms * 2; }

// column tiles of at most 72 whose part of Y^T fits the shared memory, all of one width
inline int rotate_tiles(int k, int m) {
    const long long per_block = (long long)sizeof(double) * ((k + 3) / 4) * 32;
    const int most = (int)std::max<long long>(1, std::min<long long>(9, (long long)ROT_SMEM / per_block));
    return ((m + 7) / 8 + most - 1) / most;
}

template <bool AL>
unsigned rotate_pick(dft_context* ctx, const double* in, const double* in2, long long ldi, int k1, int k,
                     const double* Y, int m, double* out, long long ldo, long long n, double alpha, double beta,
                     double* ss) {
    const int tiles = rotate_tiles(k, m);
    const int rj = ((m + tiles - 1) / tiles + 7) / 8;
#define DFT_ROT(R, P) return rotate_launch<R, P, AL>(ctx, in, in2, ldi, k1, k, Y, m, out, ldo, n, alpha, beta, ss)
    switch (rj) {
        case 1:
            // one step of few rows: more points per warp keep more loads in flight (128^3, 1 -> 1 41 -> 37 us, 3 -> 3
            // 50 -> 42; no gain from 4 rows on)
            if (k <= 3) DFT_ROT(1, 4);
            DFT_ROT(1, 2);
        case 2: DFT_ROT(2, 2);
        case 3: DFT_ROT(3, 1);
        case 4: DFT_ROT(4, 1);
        case 5: DFT_ROT(5, 1);
        case 6: DFT_ROT(6, 1);
        case 7: DFT_ROT(7, 1);
        case 8: DFT_ROT(8, 1);
        default: DFT_ROT(9, 1);
    }
#undef DFT_ROT
}

}  // namespace

bool rotate_in_place(int k, int m) { return rotate_tiles(k, m) == 1; }

// out = beta*out + alpha * in * Y   (Y: k x m host row-major)
void rotate(dft_context* ctx, const Grid& g, const double* in, long long ldi, int k, const std::vector<double>& Y, int m,
            double* out, long long ldo, double alpha, double beta) {
    if (m == 0) return;
    if (k == 0) {
        if (beta == 0.0)
            for (int j = 0; j < m; ++j)
                DFT_CUDA(cudaMemsetAsync(out + (long long)j * ldo, 0, sizeof(double) * (size_t)g.N, ctx->stream));
        return;
    }
    if (k > 1600) fail(DFT_INVALID_ARGUMENT, "subspace too large for the rotation kernel (k=%d)", k);
    double* dy = (double*)ws_get(ctx, WS_TMP, sizeof(double) * (size_t)k * m);
    DFT_CUDA(cudaMemcpyAsync(dy, Y.data(), sizeof(double) * (size_t)k * m, cudaMemcpyHostToDevice, ctx->stream));
    if (aligned16(in, ldi) && aligned16(out, ldo))
        rotate_pick<true>(ctx, in, in, ldi, k, k, dy, m, out, ldo, g.N, alpha, beta, nullptr);
    else
        rotate_pick<false>(ctx, in, in, ldi, k, k, dy, m, out, ldo, g.N, alpha, beta, nullptr);
}

namespace {

template <int RJ, int PP, bool AL>
unsigned residual_launch(dft_context* ctx, const double* AV, const double* V, long long ld, int k, const double* Y,
                         const double* theta, int m, double* R, long long n, double* ss) {
    const size_t smem = sizeof(double) * (size_t)((k + 3) / 4) * RJ * 32;
    if (smem > 32 * 1024)
        DFT_CUDA(cudaFuncSetAttribute(residual_mma_kernel<RJ, PP, AL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)ROT_SMEM));
    const int threads = smem > 90 * 1024 ? 512 : 256;
    const long long warps_needed = (n + 16 * PP - 1) / (16 * PP), resident = (long long)ctx->num_sms * 512 / threads;
    const long long bx = std::max<long long>(1, std::min<long long>((warps_needed * 32 + threads - 1) / threads, resident));
    residual_mma_kernel<RJ, PP, AL><<<(unsigned)bx, threads, smem, ctx->stream>>>(AV, V, ld, k, Y, theta, m, R, n, ss);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    return (unsigned)bx;
}

template <bool AL>
unsigned residual_pick(dft_context* ctx, const double* AV, const double* V, long long ld, int k, const double* Y,
                       const double* theta, int m, double* R, long long n, double* ss) {
    switch ((m + 7) / 8) {
        case 1: return residual_launch<1, 2, AL>(ctx, AV, V, ld, k, Y, theta, m, R, n, ss);
        case 2: return residual_launch<2, 1, AL>(ctx, AV, V, ld, k, Y, theta, m, R, n, ss);
        case 3: return residual_launch<3, 1, AL>(ctx, AV, V, ld, k, Y, theta, m, R, n, ss);
        default: return residual_launch<4, 1, AL>(ctx, AV, V, ld, k, Y, theta, m, R, n, ss);
    }
}

}  // namespace

// R_b = sum_i AV_i Y[i][b] - theta_b sum_i V_i Y[i][b] and ss[b] = sum_p R_b[p]^2 (host; synchronises):
// V Y and (AV) Y are not stored.  Up to 32 columns keep the two sums apart; wider blocks, whose
// accumulators would not fit, run as one rotation of the 2k rows [AV; V] by [Y; -Y diag(theta)].
void ritz_residual(dft_context* ctx, const Grid& g, const double* V, const double* AV, long long ld, int k,
                   const std::vector<double>& Y, const double* theta, int m, double* R, double* ss_host) {
    if (k > 1600) fail(DFT_INVALID_ARGUMENT, "subspace too large for the rotation kernel (k=%d)", k);
    const size_t nel = (size_t)k * m;
    const bool apart = m <= 32 && rotate_tiles(k, m) == 1;
    std::vector<double> Z(apart ? nel + m : 2 * nel);
    std::copy(Y.begin(), Y.begin() + nel, Z.begin());
    if (apart)
        std::copy(theta, theta + m, Z.begin() + nel);
    else
        for (int i = 0; i < k; ++i)
            for (int b = 0; b < m; ++b) Z[nel + (size_t)i * m + b] = -theta[b] * Y[(size_t)i * m + b];
    double* dz = (double*)ws_get(ctx, WS_TMP, sizeof(double) * Z.size());
    const size_t mb = rotate_max_blocks(ctx);
    double* part = (double*)ws_get(ctx, WS_REDUCE, sizeof(double) * (mb * m + m));
    double* sum = part + mb * m;
    DFT_CUDA(cudaMemcpyAsync(dz, Z.data(), sizeof(double) * Z.size(), cudaMemcpyHostToDevice, ctx->stream));
    const bool al = aligned16(V, ld) && aligned16(AV, ld) && aligned16(R, ld);
    unsigned bx;
    if (apart)
        bx = al ? residual_pick<true>(ctx, AV, V, ld, k, dz, dz + nel, m, R, g.N, part)
                : residual_pick<false>(ctx, AV, V, ld, k, dz, dz + nel, m, R, g.N, part);
    else
        bx = al ? rotate_pick<true>(ctx, AV, V, ld, k, 2 * k, dz, m, R, ld, g.N, 1.0, 0.0, part)
                : rotate_pick<false>(ctx, AV, V, ld, k, 2 * k, dz, m, R, ld, g.N, 1.0, 0.0, part);
    row_sum_kernel<<<m, 128, 0, ctx->stream>>>((int)bx, part, sum);
    DFT_LAUNCH_CHECK();
    count_launch(ctx);
    double* h = pinned(ctx, m);
    DFT_CUDA(cudaMemcpyAsync(h, sum, sizeof(double) * m, cudaMemcpyDeviceToHost, ctx->stream));
    sync(ctx);
    for (int b = 0; b < m; ++b) ss_host[b] = h[b];
}

}  // namespace dftb
