// k-bin x Legendre reductions over half spectra (the power-spectrum binning pass) and
// the per-shell Fisher-row contraction.  FP64 accumulation, deterministic two-pass sums.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "pb_common.cuh"

namespace pb {

struct RedParams {
    double edges[PB_RED_MAX_BINS + 1];
    int8_t la[PB_RED_MAX_ELLS];
    int8_t lb[PB_RED_MAX_ELLS];
    int32_t nk;
    int32_t n_ell;
};

constexpr int RED_THREADS = 256;
constexpr int RED_CHUNK = 4;  // consecutive modes per thread per step (same kz line, mostly same bin)

static int red_blocks(const Grid &G) {
    int64_t per_block = (int64_t)RED_THREADS * RED_CHUNK;
    int64_t b = (G.nhalf + per_block - 1) / per_block;
    int64_t cap = (int64_t)num_sms() * 2;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, cap));
}

// bin b with edges[b] <= k < edges[b+1], or -1
__device__ __forceinline__ int find_bin(const double *edges, int nk, double k) {
    if (!(edges[0] <= k) || !(k < edges[nk])) return -1;
    int lo = 0, hi = nk;  // invariant: edges[lo] <= k < edges[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (edges[mid] <= k) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(RED_THREADS) binred_kernel(Grid g, const typename cplx<T>::type *a,
                                                            const typename cplx<T>::type *b, const T *w,
                                                            int64_t row_stride, RedParams p, double *partials) {
    using C = typename cplx<T>::type;
    __shared__ double acc[PB_RED_MAX_ELLS * PB_RED_MAX_BINS];
    __shared__ double edges[PB_RED_MAX_BINS + 1];
    const int nk = p.nk, ne = p.n_ell;
    for (int i = threadIdx.x; i < ne * nk; i += blockDim.x) acc[i] = 0.0;
    for (int i = threadIdx.x; i <= nk; i += blockDim.x) edges[i] = p.edges[i];
    __syncthreads();
    const int row = blockIdx.y;
    const C *arow = (MODE == PB_RED_ABS2) ? a + (int64_t)row * row_stride : a;
    const C *brow = (MODE == PB_RED_CROSS) ? b + (int64_t)row * row_stride : nullptr;
    const int64_t step = (int64_t)gridDim.x * blockDim.x * RED_CHUNK;
    for (int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * RED_CHUNK; base < g.nhalf;
         base += step) {
        int cur = -1;
        double run[PB_RED_MAX_ELLS];
#pragma unroll
        for (int e = 0; e < PB_RED_MAX_ELLS; ++e) run[e] = 0.0;
        const int64_t end = min(base + RED_CHUNK, g.nhalf);
        for (int64_t idx = base; idx < end; ++idx) {
            Mode md = mode_of(g, idx);
            int bin = find_bin(edges, nk, md.k);
            if (bin != cur) {
                if (cur >= 0) {
#pragma unroll
                    for (int e = 0; e < PB_RED_MAX_ELLS; ++e)
                        if (e < ne) atomicAdd(&acc[e * nk + cur], run[e]);
                }
#pragma unroll
                for (int e = 0; e < PB_RED_MAX_ELLS; ++e) run[e] = 0.0;
                cur = bin;
            }
            if (bin < 0) continue;
            double f;
            if (MODE == PB_RED_ABS2) {
                C v = arow[idx];
                f = (double)v.x * (double)v.x + (double)v.y * (double)v.y;
            } else if (MODE == PB_RED_CROSS) {
                C u = arow[idx], v = brow[idx];
                f = (double)u.x * (double)v.x + (double)u.y * (double)v.y;
            } else {
                double v = w ? (double)w[idx] : 1.0;
                f = v * v;
            }
            f *= md.deg;
#pragma unroll
            for (int e = 0; e < PB_RED_MAX_ELLS; ++e)
                if (e < ne) run[e] += f * legendre(p.la[e], md.mu) * legendre(p.lb[e], md.mu);
        }
        if (cur >= 0) {
#pragma unroll
            for (int e = 0; e < PB_RED_MAX_ELLS; ++e)
                if (e < ne) atomicAdd(&acc[e * nk + cur], run[e]);
        }
    }
    __syncthreads();
    double *dst = partials + ((int64_t)row * gridDim.x + blockIdx.x) * (ne * nk);
    for (int i = threadIdx.x; i < ne * nk; i += blockDim.x) dst[i] = acc[i];
}

// Many rows over the same modes (the Fisher rows: CROSS of one spectrum with N_bins Q rows,
// or ABS2 of a batch).  The mode geometry -- bin, degeneracy x Legendre weights, the shared
// spectrum a -- is computed once per tile of modes into shared memory and then used by every
// row of the group, instead of once per row: the FP64 |k|, mu, bin search and Legendre
// polynomials no longer scale with the row count, and each row is one streaming read.
constexpr int RR_TILE = 512;                 // modes per tile (2 per thread)
constexpr int RR_PER = RR_TILE / RED_THREADS;
constexpr int RR_ACC_DOUBLES = 6144;         // shared accumulators per block (48 KB)
constexpr int RR_RB = 8;                     // rows loaded ahead per thread

// accumulator doubles rounded up to an even count, so the double2 tile after them is aligned
__host__ __device__ __forceinline__ size_t rr_acc_len(int rows, int ne, int nk) {
    return ((size_t)rows * ne * nk + 1) & ~(size_t)1;
}

template <typename T, int MODE>
__global__ void __launch_bounds__(RED_THREADS) binred_rows_kernel(Grid g, const typename cplx<T>::type *a,
                                                                 const typename cplx<T>::type *b,
                                                                 int64_t row_stride, RedParams p, int n_rows,
                                                                 int rows_per_group, double *partials) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char rr_smem[];
    const int nk = p.nk, ne = p.n_ell;
    const int r0 = blockIdx.y * rows_per_group;
    const int nr = min(rows_per_group, n_rows - r0);
    double *acc = reinterpret_cast<double *>(rr_smem);          // [nr][ne][nk]
    double *wt = acc + rr_acc_len(rows_per_group, ne, nk);       // [ne][RR_TILE]
    double2 *as = reinterpret_cast<double2 *>(wt + (size_t)ne * RR_TILE);  // [RR_TILE] (CROSS)
    int *bins = reinterpret_cast<int *>(as + RR_TILE);            // [RR_TILE]
    __shared__ double edges[PB_RED_MAX_BINS + 1];
    for (int i = threadIdx.x; i < nr * ne * nk; i += blockDim.x) acc[i] = 0.0;
    for (int i = threadIdx.x; i <= nk; i += blockDim.x) edges[i] = p.edges[i];
    const int64_t n_tiles = (g.nhalf + RR_TILE - 1) / RR_TILE;
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t t0 = tile * RR_TILE;
        __syncthreads();  // previous tile's readers are done (and the set-up above is visible)
        for (int j = threadIdx.x; j < RR_TILE; j += blockDim.x) {
            const int64_t idx = t0 + j;
            int bin = -1;
            if (idx < g.nhalf) {
                const Mode md = mode_of(g, idx);
                bin = find_bin(edges, nk, md.k);
                if (bin >= 0) {
#pragma unroll
                    for (int e = 0; e < PB_RED_MAX_ELLS; ++e)
                        if (e < ne) wt[e * RR_TILE + j] = md.deg * legendre(p.la[e], md.mu) * legendre(p.lb[e], md.mu);
                }
                if (MODE == PB_RED_CROSS) {
                    const C v = a[idx];
                    as[j] = make_double2((double)v.x, (double)v.y);
                }
            }
            bins[j] = bin;
        }
        __syncthreads();
        // lane <-> consecutive mode (coalesced row reads).  Consecutive modes mostly share a
        // bin, so a warp first sums each contiguous run of equal bins with a segmented
        // shuffle reduction and only the run's first lane adds to shared memory: one atomic
        // per run and Legendre order instead of one per mode on the same address.
        const int lane = threadIdx.x & 31;
        for (int pass = 0; pass < RR_PER; ++pass) {
            const int j = pass * RED_THREADS + threadIdx.x;
            const int bin = bins[j];
            const bool head = lane == 0 || bins[j - 1] != bin;
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            const int seg = __popc(heads & (0xffffffffu >> (31 - lane)));  // run index of this lane
            unsigned same = 0;                                              // bit k: lane + 2^k in my run
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int o = 1 << k;
                const int sg = __shfl_down_sync(0xffffffffu, seg, o);
                if (lane + o < 32 && sg == seg) same |= 1u << k;
            }
            double2 u = make_double2(0.0, 0.0);
            if (MODE == PB_RED_CROSS && bin >= 0) u = as[j];
            double w[PB_RED_MAX_ELLS];
#pragma unroll
            for (int e = 0; e < PB_RED_MAX_ELLS; ++e) w[e] = (e < ne && bin >= 0) ? wt[e * RR_TILE + j] : 0.0;
            // RR_RB rows' values are loaded before any of them is reduced, so each thread
            // keeps RR_RB independent reads in flight
            const C *src = (MODE == PB_RED_CROSS) ? b : a;
            for (int rb = 0; rb < nr; rb += RR_RB) {
                C vals[RR_RB];
#pragma unroll
                for (int q = 0; q < RR_RB; ++q) {
                    vals[q].x = 0;
                    vals[q].y = 0;
                    if (bin >= 0 && rb + q < nr) vals[q] = src[(int64_t)(r0 + rb + q) * row_stride + t0 + j];
                }
#pragma unroll
                for (int q = 0; q < RR_RB; ++q) {
                    if (rb + q >= nr) break;
                    double f;
                    if (MODE == PB_RED_CROSS) f = u.x * (double)vals[q].x + u.y * (double)vals[q].y;
                    else f = (double)vals[q].x * (double)vals[q].x + (double)vals[q].y * (double)vals[q].y;
                    double *accr = acc + (size_t)(rb + q) * ne * nk;
#pragma unroll
                    for (int e = 0; e < PB_RED_MAX_ELLS; ++e) {
                        if (e >= ne) break;
                        double v = f * w[e];
#pragma unroll
                        for (int k = 0; k < 5; ++k) {
                            const double up = __shfl_down_sync(0xffffffffu, v, 1 << k);
                            if (same & (1u << k)) v += up;
                        }
                        if (head && bin >= 0) atomicAdd(&accr[e * nk + bin], v);
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int r = 0; r < nr; ++r) {
        double *dst = partials + ((int64_t)(r0 + r) * gridDim.x + blockIdx.x) * (ne * nk);
        for (int i = threadIdx.x; i < ne * nk; i += blockDim.x) dst[i] = acc[(size_t)r * ne * nk + i];
    }
}

// bin (-1: none) and deg L_la L_lb of every mode, tabulated once per call for the many-row kernels
template <typename B>
__global__ void binred_geom_kernel(Grid g, RedParams p, B *mbin, double *mw) {
    __shared__ double edges[PB_RED_MAX_BINS + 1];
    for (int i = threadIdx.x; i <= p.nk; i += blockDim.x) edges[i] = p.edges[i];
    __syncthreads();
    const int ne = p.n_ell;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < g.nhalf;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const Mode md = mode_of(g, idx);
        const int bin = find_bin(edges, p.nk, md.k);
        mbin[idx] = (B)bin;
        if (bin >= 0) {
#pragma unroll
            for (int e = 0; e < PB_RED_MAX_ELLS; ++e)
                if (e < ne) mw[idx * ne + e] = md.deg * legendre(p.la[e], md.mu) * legendre(p.lb[e], md.mu);
        }
    }
}

// ------------------------------------------------------------------------------------
// Many FP64 rows, staged: a block owns up to 32 rows and walks the binned runs of its kz lines in
// segments of 16 modes.  The rows' values arrive in shared memory by cp.async, 256 contiguous bytes
// per row and two segments ahead, the segment's geometry (tabulated by binred_geom_kernel) and the
// shared spectrum beside them; a lane owns one row (odd row stride: no bank conflicts) and the
// multipoles of its warp's share, keeps the sums of the current bin in registers and adds
// them to its own slot of the block's accumulators [bin][e][row] when the bin changes: no
// atomics, a fixed order.  Streaming from memory bounds it; the lane-per-row kernel below read each
// row by one lane, 64 bytes at a time with 11 warps per SM.  (Computing the geometry in a warp of its
// own instead of reading the table took 375 us: its sqrt, search and Legendre chain per segment was longer
// than everything else.)
// Measured on a B200, 60 rows of 128^3, 20 bins, l = 0, 2, 4: 193 us against 450 us
// for the lane-per-row kernel (finalize and table included; 120 rows, 40 bins 497 against 1130 us; 203 rows, 12 bins,
// l = 0 307 against 690 us; the two tie at 64^3).
// ------------------------------------------------------------------------------------
constexpr int RT_SEG = 16;        // modes per segment
constexpr int RT_STAGES = 3;
constexpr int RT_ROWS = 32;       // rows per block (64 a block took 226 against 193 us)
constexpr int RT_LD = RT_SEG + 1;
constexpr int RT_SMEM = 220 * 1024;
// warps of a block: groups of multipoles (one or two per thread) times parts of a segment (with one or
// two multipoles, so that the block still has four warps)
__host__ __device__ constexpr int rt_egroups(int ne) { return ne <= 4 ? ne : (ne + 1) / 2; }
__host__ __device__ constexpr int rt_parts(int ne) { return ne == 1 ? 4 : ne == 2 ? 2 : 1; }
__host__ __device__ constexpr int rt_warps(int ne) { return rt_egroups(ne) * rt_parts(ne); }

__device__ __forceinline__ void rt_copy16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}

template <int BYTES> __device__ __forceinline__ void rt_copy(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES));
}

__host__ __device__ constexpr size_t rt_smem(int nk, int ne) {
    constexpr int RB = RT_ROWS;
    return (size_t)RT_STAGES * ((size_t)RB * RT_LD * 16 + RT_SEG * 16 + (size_t)ne * RT_SEG * 8 + RT_SEG * 4) +
           (size_t)rt_parts(ne) * nk * ne * RB * 8;
}

// the next segment of the block's lines: first mode and count (0: done)
struct RtWalk {
    int line, step, n_lines, l, l_end;
    float fx, fy, lo2, hi2;
    __device__ __forceinline__ int next(const Grid &g, int64_t &first) {
        while (l >= l_end) {
            line += step;
            if (line >= n_lines) return 0;
            // the run of the line that may hold binned modes, in units of kf2; FP32 with a margin for its rounding on
            // the squares (lo^2 - r^2 may be small beside both where kf0 or kf1 is far above kf2) and two modes each
            // side (the bins of the table decide)
            const int i = (int)((uint32_t)line / (uint32_t)g.n1), j = (int)line - i * g.n1;
            const float kx = freq_index(i, g.n0) * fx, ky = freq_index(j, g.n1) * fy;
            const float r2 = kx * kx + ky * ky, h2 = hi2 * (1.0f + 1e-5f) - r2;
            if (h2 < 0.0f) continue;
            const float l2 = lo2 * (1.0f - 1e-5f) - r2;
            l = l2 > 0.0f ? max(0, (int)sqrtf(l2) - 2) : 0;
            l_end = (int)fminf((float)g.nh2, sqrtf(h2) + 3.0f);
        }
        first = (int64_t)line * g.nh2 + l;
        const int c = min(RT_SEG, l_end - l);
        l += c;
        return c;
    }
};

template <int MODE, int NE>
__global__ void __launch_bounds__(32 * rt_warps(NE)) binred_tile_kernel(Grid g, const double2 *a, const double2 *b,
                                                                 int64_t row_stride, int n_rows, int nk, float lo,
                                                                 float hi, const int32_t *mbin, const double *mw,
                                                                 double *partials) {
    constexpr int RB = RT_ROWS, EG = rt_egroups(NE), EP = (NE + EG - 1) / EG, MS = rt_parts(NE);
    constexpr int NW = rt_warps(NE), NT = 32 * NW, PART = RT_SEG / MS;
    extern __shared__ __align__(16) unsigned char rt_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double2 *const rows = reinterpret_cast<double2 *>(rt_raw);                    // [stage][RB][RT_LD]
    double2 *const as = rows + (size_t)RT_STAGES * RB * RT_LD;                    // [stage][RT_SEG]
    double *const wt = reinterpret_cast<double *>(as + RT_STAGES * RT_SEG);       // [stage][RT_SEG][NE]
    double *const acc = wt + RT_STAGES * NE * RT_SEG;                             // [part][bin][e][RB]
    int *const bins = reinterpret_cast<int *>(acc + (size_t)MS * nk * NE * RB);   // [stage][RT_SEG]
    const int r0 = blockIdx.y * RB, nr = min(RB, n_rows - r0);
    const double2 *const src = (MODE == PB_RED_CROSS ? b : a) + (int64_t)r0 * row_stride;
    for (int i = threadIdx.x; i < MS * nk * NE * RB; i += NT) acc[i] = 0.0;
    const float inv = 1.0f / (float)g.kf2;
    RtWalk walk{(int)blockIdx.x - (int)gridDim.x, (int)gridDim.x, g.n0 * g.n1, 0, 0,
                (float)g.kf0 * inv, (float)g.kf1 * inv, lo > 0.0f ? lo * lo * inv * inv : 0.0f, hi * hi * inv * inv};
    int count[RT_STAGES];  // of the segments in flight (every thread walks alike)
    auto issue = [&](int st) -> int {
        int64_t first = 0;
        const int c = walk.next(g, first);
        // half a warp per row: 256 contiguous bytes
        const int m = lane & (RT_SEG - 1);
        if (m < c) {
            double2 *dst = rows + (size_t)st * RB * RT_LD + m;
            const double2 *from = src + first + m;
            for (int r = 2 * warp + (lane >> 4); r < nr; r += 2 * NW) rt_copy16(dst + r * RT_LD, from + (int64_t)r * row_stride);
            if (MODE == PB_RED_CROSS && warp == NW - 1 && lane < RT_SEG) rt_copy16(as + st * RT_SEG + m, a + first + m);
            if (warp == NW - 1 && lane >= RT_SEG) rt_copy<4>(bins + st * RT_SEG + m, mbin + first + m);
        }
        if (threadIdx.x < c * NE) rt_copy<8>(wt + st * RT_SEG * NE + threadIdx.x, mw + first * NE + threadIdx.x);
        asm volatile("cp.async.commit_group;\n" ::);
        return c;
    };
#pragma unroll
    for (int st = 0; st < RT_STAGES - 1; ++st) count[st] = issue(st);
    const int row = lane, eg = warp % EG, part = warp / EG;
    const bool mine = row < nr;
    double *const own = acc + (size_t)part * nk * NE * RB + row;
    double sum[EP];
#pragma unroll
    for (int k = 0; k < EP; ++k) sum[k] = 0.0;
    int cur = -1;
    auto flush = [&]() {
#pragma unroll
        for (int k = 0; k < EP; ++k) {
            const int e = eg + k * EG;
            if (cur >= 0 && e < NE) own[((size_t)cur * NE + e) * RB] += sum[k];
            sum[k] = 0.0;
        }
    };
    bool more = true;
    while (more) {
#pragma unroll
        for (int st = 0; st < RT_STAGES; ++st) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(RT_STAGES - 2));
            __syncthreads();  // segment st is in shared memory; everyone is done with the one before it
            count[(st + RT_STAGES - 1) % RT_STAGES] = issue((st + RT_STAGES - 1) % RT_STAGES);
            const int c = count[st];
            if (c == 0) {
                more = false;
                break;
            }
            if (mine) {
                const double2 *v = rows + ((size_t)st * RB + row) * RT_LD, *u = as + st * RT_SEG;
                const double *w = wt + st * RT_SEG * NE + eg;
                const int *bn = bins + st * RT_SEG;
                const int m1 = min(c, (part + 1) * PART);
                for (int m = part * PART; m < m1; m += 4) {
                    // four modes' operands before any is used (values past c are stale, their bins skip them)
                    double f[4], ww[4][EP];
                    int bb[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        bb[q] = m + q < m1 ? bn[m + q] : -1;
                        const double2 x = v[m + q];
                        if (MODE == PB_RED_CROSS) {
                            const double2 y = u[m + q];
                            f[q] = y.x * x.x + y.y * x.y;
                        } else {
                            f[q] = x.x * x.x + x.y * x.y;
                        }
#pragma unroll
                        for (int k = 0; k < EP; ++k) ww[q][k] = eg + k * EG < NE ? w[(m + q) * NE + k * EG] : 0.0;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (bb[q] < 0) continue;
                        if (bb[q] != cur) {
                            flush();
                            cur = bb[q];
                        }
#pragma unroll
                        for (int k = 0; k < EP; ++k) sum[k] += f[q] * ww[q][k];
                    }
                }
            }
        }
    }
    if (mine) flush();
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    const int per = nk * NE;
    for (int i = threadIdx.x; i < per * nr; i += NT) {
        const int r = i / per, j = i - r * per, e = j / nk, bin = j - e * nk;
        double x = 0.0;
#pragma unroll
        for (int k = 0; k < MS; ++k) x += acc[(((size_t)k * nk + bin) * NE + e) * RB + r];
        partials[((int64_t)(r0 + r) * gridDim.x + blockIdx.x) * per + j] = x;
    }
}

struct TileLaunch {
    int gx;
    size_t smem, geom_bytes;   // bins (int32, padded to 256 bytes) and weights of every mode
};
// the staged kernel serves 16 rows and more whose accumulators fit beside the stages
static bool tile_plan(const Grid &G, int n_rows, int nk, int n_ell, TileLaunch *t) {
    if (tuning().red_method != 0 || n_rows < 16) return false;
    t->smem = rt_smem(nk, n_ell);
    if (t->smem > (size_t)RT_SMEM) return false;
    // as many blocks as are resident at once, shared among the groups of rows
    const int groups = (n_rows + RT_ROWS - 1) / RT_ROWS;
    const int per_sm = (int)std::min<size_t>(5, (225 * 1024) / (t->smem + 1024));
    t->gx = (int)std::min<int64_t>((int64_t)G.n0 * G.n1, std::max(1, (per_sm * num_sms() + groups - 1) / groups));
    t->geom_bytes = ((size_t)G.nhalf * 4 + 255) / 256 * 256 + (size_t)G.nhalf * n_ell * sizeof(double);
    return true;
}

// ------------------------------------------------------------------------------------
// Many rows, one lane per row.  The mode geometry (bin and deg x L_la L_lb per mode, FP64)
// is tabulated once per call by binred_geom_kernel.  A warp then walks kz lines of the half
// grid; each lane reads ITS row's values along the line (8 consecutive modes = one 128-byte
// segment for complex128) while the geometry and the shared spectrum are warp-uniform
// broadcasts.  All lanes see the same mode sequence, so a bin change is a uniform branch:
// the sums of the current bin stay in registers and are added to the lane's slot of the
// warp's shared-memory accumulators [bin][e][lane] only when the bin changes (no shuffles,
// no atomics, fixed order: deterministic).  Only the part of each line inside the binned
// range is read (|k| grows along a kz line, so it is one contiguous run of modes).
// ------------------------------------------------------------------------------------
constexpr int BL_MODES = 4;  // modes per lane per step (the next step's values load meanwhile)

template <typename T, int MODE, int NE>
__global__ void __launch_bounds__(256) binred_lanes_kernel(Grid g, const typename cplx<T>::type *a,
                                                           const typename cplx<T>::type *b, int64_t row_stride,
                                                           int n_rows, int nk, const int8_t *mbin, const double *mw,
                                                           double *partials) {
    using C = typename cplx<T>::type;
    constexpr int S = BL_MODES;
    extern __shared__ __align__(16) double bl_acc[];  // [warp][bin][e][32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int per = nk * NE;
    double *wacc = bl_acc + (size_t)warp * per * 32;
    for (int i = threadIdx.x; i < nw * per * 32; i += blockDim.x) bl_acc[i] = 0.0;
    __syncthreads();
    const int row = blockIdx.y * 32 + lane;
    const bool live = row < n_rows;
    const C *brow = b + (int64_t)(live ? row : 0) * row_stride;
    const int64_t n_lines = (int64_t)g.n0 * g.n1;
    const int nh2 = g.nh2;
    double r[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) r[e] = 0.0;
    int cur = -1;
    for (int64_t line = (int64_t)blockIdx.x * nw + warp; line < n_lines; line += (int64_t)gridDim.x * nw) {
        const int64_t base = line * nh2;
        // the binned run [l_lo, l_hi) of this line
        int l_lo = nh2, l_hi = 0;
        for (int l0 = 0; l0 < nh2; l0 += 32) {
            const int l = l0 + lane;
            const bool in = l < nh2 && mbin[base + l] >= 0;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (m) {
                l_lo = min(l_lo, l0 + __ffs(m) - 1);
                l_hi = l0 + 32 - __clz(m);
            }
        }
        if (l_lo >= l_hi) continue;
        // software pipeline: the row values of step s + 1 are in flight while step s is summed
        C v[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            v[k].x = 0;
            v[k].y = 0;
            if (live && l_lo + k < l_hi) v[k] = brow[base + l_lo + k];
        }
        for (int l0 = l_lo; l0 < l_hi; l0 += S) {
            C nv[S];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                nv[k].x = 0;
                nv[k].y = 0;
                if (live && l0 + S + k < l_hi) nv[k] = brow[base + l0 + S + k];
            }
            // this step's geometry and shared spectrum, loaded before any of it is used
            int bn[S];
            C av[S];
            double w[S][NE];
#pragma unroll
            for (int k = 0; k < S; ++k) {
                const int64_t idx = base + l0 + k;
                const bool in = l0 + k < l_hi;
                bn[k] = in ? (int)mbin[idx] : -2;
                if (MODE == PB_RED_CROSS) {
                    av[k].x = 0;
                    av[k].y = 0;
                    if (in) av[k] = a[idx];
                }
#pragma unroll
                for (int e = 0; e < NE; ++e) w[k][e] = in ? mw[idx * NE + e] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < S; ++k) {
                if (bn[k] == -2) break;
                if (bn[k] != cur) {
#pragma unroll
                    for (int e = 0; e < NE; ++e) {
                        if (cur >= 0) wacc[(cur * NE + e) * 32 + lane] += r[e];
                        r[e] = 0.0;
                    }
                    cur = bn[k];
                }
                if (bn[k] < 0) continue;
                double f;
                if (MODE == PB_RED_CROSS)
                    f = (double)av[k].x * (double)v[k].x + (double)av[k].y * (double)v[k].y;
                else
                    f = (double)v[k].x * (double)v[k].x + (double)v[k].y * (double)v[k].y;
#pragma unroll
                for (int e = 0; e < NE; ++e) r[e] += f * w[k][e];
            }
#pragma unroll
            for (int k = 0; k < S; ++k) v[k] = nv[k];
        }
    }
#pragma unroll
    for (int e = 0; e < NE; ++e)
        if (cur >= 0) wacc[(cur * NE + e) * 32 + lane] += r[e];
    __syncthreads();
    // warps' sums in fixed order -> this block's partial of each row
    for (int i = threadIdx.x; i < per * 32; i += blockDim.x) {
        const int ln = i & 31, be = i >> 5;  // be = bin * NE + e
        const int rr = blockIdx.y * 32 + ln;
        if (rr >= n_rows) continue;
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += bl_acc[((size_t)w * per + be) * 32 + ln];
        const int bin = be / NE, e = be - bin * NE;
        partials[((int64_t)rr * gridDim.x + blockIdx.x) * per + e * nk + bin] = s;
    }
}

// ------------------------------------------------------------------------------------
// Few rows (a field's own spectrum): the folded reduction.
//
// The mode-tile kernel spends its time on the geometry (FP64 sqrt, division, bin search and
// Legendre polynomials per mode), not on the spectrum.  Here
//  * the four modes (+-kx, +-ky, kz) share one evaluation: their |x|^2 are summed first;
//  * bins are found from s = |k|^2 against thresholds t_b, the smallest doubles with
//    sqrt(t_b) >= edge_b (sqrt is monotone and correctly rounded on both sides, so membership
//    is bit for bit that of |k|), and s grows along a lane's walk over ky, so the search is
//    one comparison with the next threshold;
//  * the Legendre products are polynomials in mu^2 = kz^2 / s, evaluated by Horner's rule (sums of f mu^(2m), turned into
//    the products once per block, made an infinite mode NaN: inf - inf, and inf mu^2 at kz = 0).
// A unit is 32 consecutive kz of a kx plane (coalesced reads) times a run of ky that one warp
// walks; each lane keeps the sums of its current bin in registers and adds them to its own slot
// of the warp's shared-memory window [bin - first bin of the unit][product][lane] when the bin
// changes; the window is summed over the lanes into the warp's totals after the unit.  No
// atomics, a fixed order.  The window holds the bins that a unit can meet (a bound from the
// bin widths), so that 16 warps fit on an SM; with all 40 bins' slots only 6 did (483 us).
// Measured on a B200, one FP32 spectrum of 512^3, 40 bins, l = 0, 2, 4: 222 us against 2450 us
// for the mode-tile kernel (256^3 FP32: 42 against 310 us; 128^3 FP64: below 20 against 50 us).
// ------------------------------------------------------------------------------------
constexpr int FOLD_MAX_M = 5;           // mu^0 .. mu^8
// Kernels are compiled for slots of one degree in mu^2 each: l = 0; 0, 2; 0, 2, 4; and the six different products of two
// of 0, 2, 4 (those of 0, 2 fit the three slots).  Equal products share a slot.
__host__ __device__ constexpr int fold_degree(int ne, int e) { return ne <= 3 || e < 3 ? e : e - 1; }
constexpr int FOLD_SMEM = 100 * 1024;   // accumulators per block, two blocks per SM

struct FoldParams {
    double t[PB_RED_MAX_BINS + 1];                  // thresholds on |k|^2
    double coef[PB_RED_MAX_ELLS][FOLD_MAX_M];       // the slots' products as polynomials in mu^2
    int32_t nk, n_ell;
    int8_t slot[PB_RED_MAX_ELLS];                   // of each requested product
    int32_t jseg, n_jseg, n_lchunk;                 // ky steps per unit, units per (kx, kz chunk)
    int32_t wb;                                     // bins of a unit's window
};

template <typename T, int MODE>
__device__ __forceinline__ double fold_value(const typename cplx<T>::type *a, const typename cplx<T>::type *b,
                                             const T *w, int64_t idx) {
    if (MODE == PB_RED_ABS2) {
        const typename cplx<T>::type v = a[idx];
        return (double)v.x * (double)v.x + (double)v.y * (double)v.y;
    }
    if (MODE == PB_RED_CROSS) {
        const typename cplx<T>::type u = a[idx], v = b[idx];
        return (double)u.x * (double)v.x + (double)u.y * (double)v.y;
    }
    const double v = w ? (double)w[idx] : 1.0;
    return v * v;
}

template <typename T, int MODE, int NE>
__global__ void __launch_bounds__(256, 2) binred_fold_kernel(Grid g, const typename cplx<T>::type *a,
                                                            const typename cplx<T>::type *b, const T *w,
                                                            int64_t row_stride, const __grid_constant__ FoldParams p,
                                                            double *partials) {
    constexpr int U = sizeof(T) == 4 ? 4 : 2;  // ky steps whose values are in flight together
    extern __shared__ __align__(16) double fold_smem[];  // [warp][window bin][product][32], [warp][bin][product]
    __shared__ double t[PB_RED_MAX_BINS + 2];
    const int nk = p.nk, nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = nk * NE, wper = p.wb * NE;
    double *const win = fold_smem + (size_t)warp * wper * 32;
    double *const totals = fold_smem + (size_t)nw * wper * 32;
    double *const tot = totals + (size_t)warp * per;
    for (int i = threadIdx.x; i < nw * (wper * 32 + per); i += blockDim.x) fold_smem[i] = 0.0;
    for (int i = threadIdx.x; i <= nk; i += blockDim.x) t[i] = p.t[i];
    if (threadIdx.x == 0) t[nk + 1] = __longlong_as_double(0x7ff0000000000000LL);
    __syncthreads();
    const int row = blockIdx.y;
    if (MODE == PB_RED_ABS2) a += (int64_t)row * row_stride;
    if (MODE == PB_RED_CROSS) b += (int64_t)row * row_stride;
    const int h0 = g.n0 >> 1, h1 = g.n1 >> 1;       // frequency f >= 0 sits at f < n / 2, f < 0 at f + n
    const int m0 = g.n0 - h0, m1 = g.n1 - h1;       // largest |f| of each axis
    const int64_t units = (int64_t)(m0 + 1) * p.n_lchunk * p.n_jseg;
    const double t_lo = p.t[0], t_hi = p.t[nk];
    for (int64_t u = (int64_t)blockIdx.x * nw + warp; u < units; u += (int64_t)gridDim.x * nw) {
        const int js = (int)(u % p.n_jseg);
        const int64_t r = u / p.n_jseg;
        const int l0 = (int)(r % p.n_lchunk) * 32, l = l0 + lane, fi = (int)(r / p.n_lchunk);
        const bool live = l < g.nh2, hp = fi < h0, hm = fi >= 1;
        const int64_t op = (int64_t)(hp ? fi : 0) * g.n1 * g.nh2 + l, om = (int64_t)(hm ? g.n0 - fi : 0) * g.n1 * g.nh2 + l;
        const double kx = __dmul_rn((double)fi, g.kf0), kz = __dmul_rn((double)l, g.kf2);
        const double kx2 = __dmul_rn(kx, kx), kz2 = __dmul_rn(kz, kz);
        const double deg = l > 0 ? 2.0 : 1.0;
        const int jb = js * p.jseg, j1 = min(jb + p.jseg, m1 + 1);
        // the unit's first bin: the one of its smallest |k|^2 (or the first edge still ahead)
        int base;
        {
            const double ky = __dmul_rn((double)jb, g.kf1), kzb = __dmul_rn((double)l0, g.kf2);
            const double sb = __dadd_rn(__dadd_rn(kx2, __dmul_rn(ky, ky)), __dmul_rn(kzb, kzb));
            if (sb >= t_hi) continue;
            base = 0;
            while (t[base + 1] <= sb) ++base;
        }
        int bin = base - 1;      // current bin (base - 1: none yet); t[bin + 1] is the next threshold
        double next = t[base], acc[NE];
#pragma unroll
        for (int e = 0; e < NE; ++e) acc[e] = 0.0;
        for (int j0 = jb; j0 < j1; j0 += U) {
            double s[U], f[U];
            bool any = false;
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int fj = j0 + q;
                const double ky = __dmul_rn((double)fj, g.kf1);
                s[q] = __dadd_rn(__dadd_rn(kx2, __dmul_rn(ky, ky)), kz2);
                const bool in = live && fj < j1 && s[q] < t_hi;
                any = any || in;
                f[q] = 0.0;
                if (in && s[q] >= t_lo) {
                    // the up to four mirrored modes; the loads of the U steps are independent
                    const int jp = fj * g.nh2, jm = (g.n1 - fj) * g.nh2;
                    if (fj < h1) {
                        if (hp) f[q] += fold_value<T, MODE>(a, b, w, op + jp);
                        if (hm) f[q] += fold_value<T, MODE>(a, b, w, om + jp);
                    }
                    if (fj >= 1) {
                        if (hp) f[q] += fold_value<T, MODE>(a, b, w, op + jm);
                        if (hm) f[q] += fold_value<T, MODE>(a, b, w, om + jm);
                    }
                }
            }
            if (!__any_sync(0xffffffffu, any)) break;  // s only grows from here
#pragma unroll
            for (int q = 0; q < U; ++q) {
                if (s[q] >= next) {
                    if (bin >= base) {
#pragma unroll
                        for (int e = 0; e < NE; ++e) win[((bin - base) * NE + e) * 32 + lane] += acc[e];
                    }
#pragma unroll
                    for (int e = 0; e < NE; ++e) acc[e] = 0.0;
                    do {
                        ++bin;
                        next = t[bin + 1];
                    } while (s[q] >= next);
                    // past the last edge, or a mode beyond the run: nothing more is added
                    if (bin >= nk || j0 + q >= j1) {
                        bin = base - 1;
                        next = t[nk + 1];
                    }
                }
                const double x = f[q] * deg, mu2 = NE > 1 && s[q] > 0.0 ? kz2 / s[q] : 0.0;
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const int d = fold_degree(NE, e);
                    double w = p.coef[e][d];
#pragma unroll
                    for (int m = FOLD_MAX_M - 2; m >= 0; --m)
                        if (m < d) w = w * mu2 + p.coef[e][m];
                    acc[e] += x * w;
                }
            }
        }
        if (bin >= base) {
#pragma unroll
            for (int e = 0; e < NE; ++e) win[((bin - base) * NE + e) * 32 + lane] += acc[e];
        }
        __syncwarp();
        // a lane sums one (bin, product) over the 32 slots (rotated: no bank conflicts), clearing them
        const int rows = min(p.wb, nk - base) * NE;
        for (int q = lane; q < rows; q += 32) {
            double x = 0.0;
#pragma unroll 16
            for (int k = 0; k < 32; ++k) x += win[q * 32 + ((lane + k) & 31)];
#pragma unroll 16
            for (int k = 0; k < 32; ++k) win[q * 32 + ((lane + k) & 31)] = 0.0;
            tot[base * NE + q] += x;
        }
        __syncwarp();
    }
    __syncthreads();
    for (int i = threadIdx.x; i < per; i += blockDim.x) {
        double x = totals[i];
        for (int k = 1; k < nw; ++k) x += totals[(size_t)k * per + i];
        totals[i] = x;
    }
    __syncthreads();
    double *dst = partials + ((int64_t)row * gridDim.x + blockIdx.x) * (p.n_ell * nk);
    for (int i = threadIdx.x; i < p.n_ell * nk; i += blockDim.x) {
        const int e = i / nk, bn = i - e * nk;
        dst[i] = totals[bn * NE + p.slot[e]];
    }
}

// smallest double t >= 0 with sqrt(t) >= e
static double sqrt_threshold(double e) {
    if (!(e > 0.0)) return 0.0;
    double t = e * e;
    while (t > 0.0 && std::sqrt(t) >= e) t = std::nextafter(t, 0.0);
    while (std::sqrt(t) < e) t = std::nextafter(t, HUGE_VAL);
    return t;
}

// Fills the fold parameters when the folded kernel takes this reduction: the global line of
// sight (mu of the four mirrored modes agrees) and even Legendre products, or monopoles alone (no mu; one
// FP64 row of 150 x 135 x 144 about another line of sight: 42 us by the mode-tile kernel, 12 us
// folded); false otherwise.
static bool fold_plan(const Grid &G, const RedParams &r, FoldParams *p, int *slots) {
    for (int e = 0; e < r.n_ell; ++e)
        if (G.los && (r.la[e] | r.lb[e])) return false;
    static const double leg[5][3] = {{1.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {-0.5, 1.5, 0.0}, {0.0, 0.0, 0.0},
                                     {0.375, -3.75, 4.375}};
    memset(p, 0, sizeof(*p));
    // the different products, each in the first free slot that holds its degree, in the smallest kernel with such slots
    for (int n : {1, 2, 3, 6}) {
        int used = 0, e = 0;
        memset(p->coef, 0, sizeof(p->coef));
        for (; e < r.n_ell; ++e) {
            const int la = std::min(r.la[e], r.lb[e]), lb = std::max(r.la[e], r.lb[e]), top = (la + lb) / 2;
            if ((la | lb) & 1) return false;
            int s = 0;
            while (s < e && !(std::min(r.la[s], r.lb[s]) == la && std::max(r.la[s], r.lb[s]) == lb)) ++s;
            if (s < e) {
                p->slot[e] = p->slot[s];
                continue;
            }
            for (s = 0; s < n && ((used >> s & 1) || fold_degree(n, s) < top);) ++s;
            if (s == n) break;
            used |= 1 << s;
            p->slot[e] = (int8_t)s;
            for (int i = 0; i <= la / 2; ++i)
                for (int j = 0; j <= lb / 2; ++j) p->coef[s][i + j] += leg[la][i] * leg[lb][j];
        }
        *slots = n;
        if (e == r.n_ell) break;
    }
    for (int i = 0; i <= r.nk; ++i) p->t[i] = sqrt_threshold(r.edges[i]);
    p->nk = r.nk;
    p->n_ell = r.n_ell;
    return true;
}

struct LanesLaunch {
    int nw, gx;
    size_t smem;
    size_t geom_bytes;   // mbin (nhalf bytes, padded to 256) + mw (nhalf * n_ell doubles)
};

// the lane-per-row kernel serves many rows with small (bins x multipoles) accumulators
static bool lanes_plan(const Grid &G, int n_rows, int nk, int n_ell, LanesLaunch *L) {
    const pb_tuning_t &tu = tuning();
    if (tu.red_method == 2) return false;
    if (n_rows < (tu.red_method == 1 ? 1 : 16)) return false;
    const size_t per_warp = (size_t)nk * n_ell * 32 * sizeof(double);
    if (per_warp > 48 * 1024) return false;
    const size_t fit = std::max<size_t>(1, (48 * 1024) / per_warp);
    L->nw = tu.red_warps > 0 ? (int)std::min<size_t>((size_t)tu.red_warps, 2 * fit) : (int)std::min<size_t>(4, fit);
    L->smem = per_warp * L->nw;
    if (L->smem > 96 * 1024) return false;
    const int64_t n_lines = (int64_t)G.n0 * G.n1;
    const int groups = (n_rows + 31) / 32;
    const int waves = tu.red_waves > 0 ? tu.red_waves : 8;
    int64_t gx = ((int64_t)waves * num_sms() + groups - 1) / groups;
    gx = std::min<int64_t>(gx, (n_lines + L->nw - 1) / L->nw);
    L->gx = (int)std::max<int64_t>(1, gx);
    L->geom_bytes = ((size_t)G.nhalf + 255) / 256 * 256 + (size_t)G.nhalf * n_ell * sizeof(double);
    return true;
}

__global__ void binred_finalize(const double *partials, int n_blocks, int per_row, int n_rows, double scale,
                                double *out, int accumulate) {
    const int t = blockIdx.x * SUM_COLS + threadIdx.x;
    const bool live = t < n_rows * per_row;
    const int row = live ? t / per_row : 0, j = t - row * per_row;
    double s = block_column_sum(partials + (int64_t)row * n_blocks * per_row + j, per_row, n_blocks, live);
    if (threadIdx.y != 0 || !live) return;
    s *= scale;
    out[t] = accumulate ? out[t] + s : s;
}

static void launch_binred_finalize(const double *partials, int n_blocks, int per_row, int n_rows, double scale,
                                   double *out, int accumulate, cudaStream_t s) {
    const int total = n_rows * per_row;
    binred_finalize<<<(total + SUM_COLS - 1) / SUM_COLS, dim3(SUM_COLS, SUM_ROWS), 0, s>>>(partials, n_blocks, per_row,
                                                                                          n_rows, scale, out, accumulate);
}

template <typename T, int MODE, int NE>
static cudaError_t fold_launch(const Grid &G, const void *a, const void *b, int n_rows, int64_t row_stride,
                               const FoldParams &p, int nb, int nw, double *partials, cudaStream_t s) {
    const size_t smem = (size_t)nw * (p.wb * 32 + p.nk) * NE * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(binred_fold_kernel<T, MODE, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    binred_fold_kernel<T, MODE, NE><<<dim3(nb, n_rows), 32 * nw, smem, s>>>(
        G, (const typename cplx<T>::type *)a, (const typename cplx<T>::type *)b, (const T *)a, row_stride, p, partials);
    return cudaSuccess;
}

// bins that an interval of |k| of length D can meet
static int bins_within(const double *edges, int nk, double D) {
    int most = 1;
    for (int i = 0, j = 0; i < nk; ++i) {
        // an interval that ends in bin j (edge j below its end) and starts in bin i
        while (j + 1 < nk && edges[j + 1] - edges[i + 1] <= D) ++j;
        most = std::max(most, j - i + 1);
    }
    return most;
}

// one folded reduction on nb blocks per row; false when its accumulators do not fit
static bool launch_fold(const Grid &G, int precision, int mode, const void *a, const void *b, int n_rows,
                        int64_t row_stride, const double *edges, FoldParams p, int slots, int nb,
                        double *partials, cudaStream_t s) {
    if (n_rows > 65535) return false;   // rows lie in gridDim.y
    const int m0 = G.n0 - G.n0 / 2, m1 = G.n1 - G.n1 / 2;
    p.n_lchunk = (G.nh2 + 31) / 32;
    // ky steps of a unit: 32, shorter while eight warps' windows do not fit or a warp gets fewer
    // than eight units (their work differs: 5 units of 64 steps a warp took 294 us at 512^3, 222 us now)
    int nw = 0;
    for (p.jseg = 32;; p.jseg /= 2) {
        const double dy = (p.jseg + 1) * G.kf1, dz = 32 * G.kf2;
        p.wb = std::min(p.nk, 1 + bins_within(edges, p.nk, std::sqrt(dy * dy + dz * dz)));
        nw = (int)std::min<size_t>(8, FOLD_SMEM / ((size_t)(p.wb * 32 + p.nk) * slots * sizeof(double)));
        const int64_t units = (int64_t)(m0 + 1) * p.n_lchunk * ((m1 + p.jseg) / p.jseg);
        if (p.jseg == 8 || (nw == 8 && units >= (int64_t)8 * nb * nw)) break;
    }
    // where a block holds one window only, its one warp is slower than the mode-tile kernel: all products up to l = 4 in 60
    // bins, FP64 weights of 64^3 (95 KB a window) 43 against 29 us, of 128^3 (58 KB) 94 against 64 us; with two warps, of
    // 200^3 (41 KB), 71 against 199 us
    if (nw < 2) return false;
    p.n_jseg = (m1 + p.jseg) / p.jseg;  // m1 + 1 frequencies |f| = 0 .. m1
    cudaError_t e = cudaSuccess;
#define PB_FOLD_M(T, MODE, NE) \
    case NE: e = fold_launch<T, MODE, NE>(G, a, b, n_rows, row_stride, p, nb, nw, partials, s); break;
#define PB_FOLD(T, MODE)                                                                                          \
    switch (slots) {                                                                                              \
        PB_FOLD_M(T, MODE, 1) PB_FOLD_M(T, MODE, 2) PB_FOLD_M(T, MODE, 3) PB_FOLD_M(T, MODE, 6)                    \
    }
    if (precision == PB_F32) {
        if (mode == PB_RED_ABS2) PB_FOLD(float, PB_RED_ABS2)
        else if (mode == PB_RED_CROSS) PB_FOLD(float, PB_RED_CROSS)
        else PB_FOLD(float, PB_RED_REAL2)
    } else {
        if (mode == PB_RED_ABS2) PB_FOLD(double, PB_RED_ABS2)
        else if (mode == PB_RED_CROSS) PB_FOLD(double, PB_RED_CROSS)
        else PB_FOLD(double, PB_RED_REAL2)
    }
#undef PB_FOLD
#undef PB_FOLD_M
    return e == cudaSuccess;
}

}  // namespace pb

using namespace pb;

extern "C" int pb_bin_reduce_workspace_size(const pb_grid_t *g, int n_rows, int nk, int n_ell, size_t *bytes) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!bytes) return fail(PB_ERR_INVALID, "bytes is NULL");
    if (n_rows < 1 || nk < 1 || n_ell < 1) return fail(PB_ERR_INVALID, "pb_bin_reduce: empty reduction");
    *bytes = (size_t)n_rows * red_blocks(G) * nk * n_ell * sizeof(double);
    TileLaunch t;
    if (tile_plan(G, n_rows, nk, n_ell, &t))
        *bytes = std::max(*bytes, t.geom_bytes + (size_t)n_rows * t.gx * nk * n_ell * sizeof(double));
    LanesLaunch L;
    if (lanes_plan(G, n_rows, nk, n_ell, &L))
        *bytes = std::max(*bytes, L.geom_bytes + (size_t)n_rows * L.gx * nk * n_ell * sizeof(double));
    return PB_OK;
}

extern "C" int pb_bin_reduce(const pb_grid_t *g, int precision, int mode, const void *a, const void *b,
                             int n_rows, int64_t row_stride, const double *edges, int nk, const int32_t *ells,
                             int n_ell, double scale, double *out, int accumulate, void *workspace,
                             size_t workspace_bytes, void *stream) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (nk < 1 || nk > PB_RED_MAX_BINS) return fail(PB_ERR_INVALID, "pb_bin_reduce: nk must be in [1, 64]");
    if (n_ell < 1 || n_ell > PB_RED_MAX_ELLS) return fail(PB_ERR_INVALID, "pb_bin_reduce: n_ell must be in [1, 9]");
    if (n_rows < 1 || n_rows > 65535) return fail(PB_ERR_INVALID, "pb_bin_reduce: n_rows must be in [1, 65535]");
    if (!edges || !ells || !out) return fail(PB_ERR_INVALID, "pb_bin_reduce: NULL argument");
    if (mode == PB_RED_ABS2 && !a) return fail(PB_ERR_INVALID, "pb_bin_reduce: ABS2 needs a");
    if (mode == PB_RED_CROSS && (!a || !b)) return fail(PB_ERR_INVALID, "pb_bin_reduce: CROSS needs a and b");
    if (mode < 0 || mode > 2) return fail(PB_ERR_INVALID, "pb_bin_reduce: bad mode");
    if (row_stride == 0) row_stride = G.nhalf;
    RedParams p;
    for (int i = 0; i <= nk; ++i) {
        p.edges[i] = edges[i];
        if (i > 0 && !(edges[i] > edges[i - 1]))
            return fail(PB_ERR_INVALID, "pb_bin_reduce: bin edges must be strictly increasing");
    }
    for (int e = 0; e < n_ell; ++e) {
        if (ells[2 * e] < 0 || ells[2 * e] > 4 || ells[2 * e + 1] < 0 || ells[2 * e + 1] > 4)
            return fail(PB_ERR_INVALID, "pb_bin_reduce: Legendre order must be in [0, 4]");
        p.la[e] = (int8_t)ells[2 * e];
        p.lb[e] = (int8_t)ells[2 * e + 1];
    }
    p.nk = nk;
    p.n_ell = n_ell;
    if (precision != PB_F32 && precision != PB_F64) return fail(PB_ERR_INVALID, "bad precision");
    int nb = red_blocks(G);
    size_t need = (size_t)n_rows * nb * nk * n_ell * sizeof(double);
    cudaStream_t s = as_stream(stream);
    TileLaunch TT;
    if (mode != PB_RED_REAL2 && precision == PB_F64 && tile_plan(G, n_rows, nk, n_ell, &TT)) {
        need = TT.geom_bytes + (size_t)n_rows * TT.gx * nk * n_ell * sizeof(double);
        if (!workspace || workspace_bytes < need)
            return fail(PB_ERR_WORKSPACE, "pb_bin_reduce: workspace too small (need " + std::to_string(need) + " bytes)");
        int32_t *mbin = (int32_t *)workspace;
        double *mw = (double *)((char *)workspace + ((size_t)G.nhalf * 4 + 255) / 256 * 256);
        double *partials = (double *)((char *)workspace + TT.geom_bytes);
        binred_geom_kernel<int32_t><<<(int)std::min<int64_t>((G.nhalf + 255) / 256, (int64_t)num_sms() * 8), 256, 0, s>>>(
            G, p, mbin, mw);
        PB_LAUNCH_CHECK("pb_bin_reduce(geometry)");
        const dim3 tgrid(TT.gx, (n_rows + RT_ROWS - 1) / RT_ROWS);
#define PB_RT_CASE(M, NE)                                                                                       \
    case NE:                                                                                                    \
        PB_CUDA(cudaFuncSetAttribute(binred_tile_kernel<M, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                     (int)TT.smem));                                                            \
        binred_tile_kernel<M, NE><<<tgrid, 32 * rt_warps(NE), TT.smem, s>>>(                                    \
            G, (const double2 *)a, (const double2 *)b, row_stride, n_rows, nk, (float)edges[0], (float)edges[nk], \
            mbin, mw, partials);                                                                                \
        break;
#define PB_RT_MODE(M)                                                                                       \
    switch (n_ell) {                                                                                        \
        PB_RT_CASE(M, 1) PB_RT_CASE(M, 2) PB_RT_CASE(M, 3) PB_RT_CASE(M, 4) PB_RT_CASE(M, 5) PB_RT_CASE(M, 6) \
        PB_RT_CASE(M, 7) PB_RT_CASE(M, 8) PB_RT_CASE(M, 9)                                                   \
    }
        if (mode == PB_RED_ABS2) PB_RT_MODE(PB_RED_ABS2)
        else PB_RT_MODE(PB_RED_CROSS)
#undef PB_RT_MODE
#undef PB_RT_CASE
        PB_LAUNCH_CHECK("pb_bin_reduce(tile)");
        launch_binred_finalize(partials, TT.gx, nk * n_ell, n_rows, scale, out, accumulate, s);
        PB_LAUNCH_CHECK("pb_bin_reduce(finalize)");
        return PB_OK;
    }
    LanesLaunch LL;
    if (mode != PB_RED_REAL2 && lanes_plan(G, n_rows, nk, n_ell, &LL)) {
        // geometry table, then one lane per row (binred_lanes_kernel)
        need = LL.geom_bytes + (size_t)n_rows * LL.gx * nk * n_ell * sizeof(double);
        if (!workspace || workspace_bytes < need)
            return fail(PB_ERR_WORKSPACE, "pb_bin_reduce: workspace too small (need " + std::to_string(need) + " bytes)");
        int8_t *mbin = (int8_t *)workspace;
        double *mw = (double *)((char *)workspace + ((size_t)G.nhalf + 255) / 256 * 256);
        double *partials = (double *)((char *)workspace + LL.geom_bytes);
        const int gg = (int)std::min<int64_t>((G.nhalf + 255) / 256, (int64_t)num_sms() * 8);
        binred_geom_kernel<int8_t><<<gg, 256, 0, s>>>(G, p, mbin, mw);
        PB_LAUNCH_CHECK("pb_bin_reduce(geometry)");
        dim3 lgrid(LL.gx, (n_rows + 31) / 32);
        const void *rows = (mode == PB_RED_CROSS) ? b : a;
#define PB_BL_LAUNCH(T, M, NE)                                                                                  \
    do {                                                                                                        \
        PB_CUDA(cudaFuncSetAttribute(binred_lanes_kernel<T, M, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)LL.smem));                                                            \
        binred_lanes_kernel<T, M, NE><<<lgrid, 32 * LL.nw, LL.smem, s>>>(G, (const cplx<T>::type *)a,          \
                                                                        (const cplx<T>::type *)rows, row_stride, \
                                                                        n_rows, nk, mbin, mw, partials);         \
    } while (0)
#define PB_BL_NE(T, M)                                        \
    switch (n_ell) {                                          \
        case 1: PB_BL_LAUNCH(T, M, 1); break;                 \
        case 2: PB_BL_LAUNCH(T, M, 2); break;                 \
        case 3: PB_BL_LAUNCH(T, M, 3); break;                 \
        case 4: PB_BL_LAUNCH(T, M, 4); break;                 \
        case 5: PB_BL_LAUNCH(T, M, 5); break;                 \
        case 6: PB_BL_LAUNCH(T, M, 6); break;                 \
        case 7: PB_BL_LAUNCH(T, M, 7); break;                 \
        case 8: PB_BL_LAUNCH(T, M, 8); break;                 \
        default: PB_BL_LAUNCH(T, M, 9); break;                \
    }
        if (precision == PB_F32) {
            if (mode == PB_RED_ABS2) PB_BL_NE(float, PB_RED_ABS2)
            else PB_BL_NE(float, PB_RED_CROSS)
        } else {
            if (mode == PB_RED_ABS2) PB_BL_NE(double, PB_RED_ABS2)
            else PB_BL_NE(double, PB_RED_CROSS)
        }
#undef PB_BL_NE
#undef PB_BL_LAUNCH
        PB_LAUNCH_CHECK("pb_bin_reduce(lanes)");
        launch_binred_finalize(partials, LL.gx, nk * n_ell, n_rows, scale, out, accumulate, s);
        PB_LAUNCH_CHECK("pb_bin_reduce(finalize)");
        return PB_OK;
    }
    if (!workspace || workspace_bytes < need)
        return fail(PB_ERR_WORKSPACE, "pb_bin_reduce: workspace too small (need " + std::to_string(need) + " bytes)");
    double *partials = (double *)workspace;
    // the folded kernel wherever its symmetry holds: at 128^3 FP64 CROSS, l = 0, 2, 4, it takes
    // 37 / 71 / 141 us for 4 / 8 / 15 rows against 87 / 129 / 216 us for the mode-tile kernel (from
    // 16 rows the lane-per-row kernel above takes over)
    FoldParams fp;
    int slots = 0;
    if (tuning().red_method != 2 && fold_plan(G, p, &fp, &slots) &&
        launch_fold(G, precision, mode, a, b, n_rows, row_stride, p.edges, fp, slots, nb, partials, s)) {
        PB_LAUNCH_CHECK("pb_bin_reduce(fold)");
        launch_binred_finalize(partials, nb, nk * n_ell, n_rows, scale, out, accumulate, s);
        PB_LAUNCH_CHECK("pb_bin_reduce(finalize)");
        return PB_OK;
    }
    if (mode != PB_RED_REAL2) {
        // spectra: mode geometry once per tile for a group of rows (binred_rows_kernel)
        const int per = nk * n_ell;
        const int rpg = std::max(1, std::min(n_rows, RR_ACC_DOUBLES / per));
        const size_t smem = rr_acc_len(rpg, n_ell, nk) * sizeof(double) + (size_t)n_ell * RR_TILE * sizeof(double) +
                            (size_t)RR_TILE * (sizeof(double2) + sizeof(int));
        dim3 rgrid(nb, (n_rows + rpg - 1) / rpg);
#define PB_RR_LAUNCH(T, M)                                                                                   \
    do {                                                                                                     \
        PB_CUDA(cudaFuncSetAttribute(binred_rows_kernel<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)smem));                                                            \
        binred_rows_kernel<T, M><<<rgrid, RED_THREADS, smem, s>>>(G, (const cplx<T>::type *)a,              \
                                                                  (const cplx<T>::type *)b, row_stride, p,   \
                                                                  n_rows, rpg, partials);                    \
    } while (0)
        if (precision == PB_F32) {
            if (mode == PB_RED_ABS2) PB_RR_LAUNCH(float, PB_RED_ABS2);
            else PB_RR_LAUNCH(float, PB_RED_CROSS);
        } else if (precision == PB_F64) {
            if (mode == PB_RED_ABS2) PB_RR_LAUNCH(double, PB_RED_ABS2);
            else PB_RR_LAUNCH(double, PB_RED_CROSS);
        } else {
            return fail(PB_ERR_INVALID, "bad precision");
        }
#undef PB_RR_LAUNCH
        PB_LAUNCH_CHECK("pb_bin_reduce(rows)");
        launch_binred_finalize(partials, nb, per, n_rows, scale, out, accumulate, s);
        PB_LAUNCH_CHECK("pb_bin_reduce(finalize)");
        return PB_OK;
    }
    dim3 grid(nb, n_rows);
#define PB_RED_LAUNCH(T, M)                                                                        \
    binred_kernel<T, M><<<grid, RED_THREADS, 0, s>>>(G, (const cplx<T>::type *)a, (const cplx<T>::type *)b, \
                                                      (const T *)a, row_stride, p, partials)
    if (precision == PB_F32) {
        if (mode == PB_RED_ABS2) PB_RED_LAUNCH(float, PB_RED_ABS2);
        else if (mode == PB_RED_CROSS) PB_RED_LAUNCH(float, PB_RED_CROSS);
        else PB_RED_LAUNCH(float, PB_RED_REAL2);
    } else if (precision == PB_F64) {
        if (mode == PB_RED_ABS2) PB_RED_LAUNCH(double, PB_RED_ABS2);
        else if (mode == PB_RED_CROSS) PB_RED_LAUNCH(double, PB_RED_CROSS);
        else PB_RED_LAUNCH(double, PB_RED_REAL2);
    } else {
        return fail(PB_ERR_INVALID, "bad precision");
    }
#undef PB_RED_LAUNCH
    PB_LAUNCH_CHECK("pb_bin_reduce");
    launch_binred_finalize(partials, nb, nk * n_ell, n_rows, scale, out, accumulate, s);
    PB_LAUNCH_CHECK("pb_bin_reduce(finalize)");
    return PB_OK;
}

// ------------------------------------------------------------------------------------
// Fisher rows over one k-shell:  out[orow[r]][j] = scale * sum_{i} deg_i Re(conj(F[key_r](m_i)) Q_j(m_i))
// over the shell's mode list m_i: a dense product of <= 32 rows with all columns, FP64.  A block owns
// 8 RPT rows and 64 columns and walks its part of the list 16 modes at a time: the next modes' values
// (gathered, runs of kz) load into registers while the current ones, staged in shared memory with an
// odd row stride, feed RPT x 4 sums per thread.  One partial per block, summed in order by a second
// pass.  Reading Q (each mode once per group of rows) bounds it.  The kernel before took one
// sum per shared-memory pair and wrote a partial every 32 modes: 90 us a shell of 17 rows, 203
// columns and 37,000 modes at 128^3 (and 11 us to sum the partials) against 56 us.
// ------------------------------------------------------------------------------------
namespace pb {
constexpr int SR_THREADS = 128;
constexpr int SR_M = 16;    // modes per step
constexpr int SR_R = 32;    // rows per launch
constexpr int SR_CT = 64;   // columns per block

struct ShellRowKeys {
    int32_t key[SR_R];
};

template <typename T, int RPT>
__global__ void __launch_bounds__(SR_THREADS) shell_rows_kernel(Grid g, const typename cplx<T>::type *F,
                                                               const typename cplx<T>::type *Q, int n_rows,
                                                               int n_cols, const int64_t *modes, int64_t n_modes,
                                                               int64_t per_block, ShellRowKeys keys, double *partials) {
    using C = typename cplx<T>::type;
    constexpr int NR = 8 * RPT, FL = NR * SR_M / SR_THREADS, QL = SR_CT * SR_M / SR_THREADS;
    __shared__ double2 Fs[NR][SR_M + 1];
    __shared__ double2 Qs[SR_CT][SR_M + 1];
    const int tid = threadIdx.x, m = tid & (SR_M - 1), h = tid / SR_M;   // loads: mode m of rows h, h + 8, ...
    const int tx = tid & 15, ty = tid >> 4;                              // sums: columns tx + 16 c, rows ty + 8 r
    const int j0 = blockIdx.y * SR_CT;
    const int64_t i0 = (int64_t)blockIdx.x * per_block, i1 = min(i0 + per_block, n_modes);
    double acc[RPT][4];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
    C f[FL], q[QL];
    double deg = 0.0;
    // this thread's mode of the step from i, -1 past the end
    auto mode_at = [&](int64_t i) -> int64_t { return i + m < i1 ? modes[i + m] : -1; };
    auto fetch = [&](int64_t idx) {
        deg = (uint64_t)idx % (uint64_t)g.nh2 > 0 ? 2.0 : 1.0;
#pragma unroll
        for (int k = 0; k < FL; ++k) {
            const int r = h + 8 * k;
            f[k].x = f[k].y = 0;
            if (idx >= 0 && r < n_rows) f[k] = F[(int64_t)keys.key[r] * g.nhalf + idx];
        }
#pragma unroll
        for (int k = 0; k < QL; ++k) {
            const int j = j0 + h + 8 * k;
            q[k].x = q[k].y = 0;
            if (idx >= 0 && j < n_cols) q[k] = Q[(int64_t)j * g.nhalf + idx];
        }
    };
    int64_t next = mode_at(i0);
    fetch(next);
    next = mode_at(i0 + SR_M);
    for (int64_t i = i0; i < i1; i += SR_M) {
        __syncthreads();  // the step before has been used
#pragma unroll
        for (int k = 0; k < FL; ++k) Fs[h + 8 * k][m] = make_double2(deg * (double)f[k].x, deg * (double)f[k].y);
#pragma unroll
        for (int k = 0; k < QL; ++k) Qs[h + 8 * k][m] = make_double2((double)q[k].x, (double)q[k].y);
        __syncthreads();
        if (i + SR_M < i1) {
            fetch(next);
            next = mode_at(i + 2 * SR_M);
        }
#pragma unroll 4
        for (int k = 0; k < SR_M; ++k) {
            double2 a[RPT], b[4];
#pragma unroll
            for (int r = 0; r < RPT; ++r) a[r] = Fs[ty + 8 * r][k];
#pragma unroll
            for (int c = 0; c < 4; ++c) b[c] = Qs[tx + 16 * c][k];
#pragma unroll
            for (int r = 0; r < RPT; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] += a[r].x * b[c].x + a[r].y * b[c].y;
        }
    }
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int row = ty + 8 * r, col = j0 + tx + 16 * c;
            if (row < n_rows && col < n_cols) partials[((int64_t)blockIdx.x * n_rows + row) * n_cols + col] = acc[r][c];
        }
}

// parts of the mode list: enough blocks for three per SM, down to one step each.  A step is a chain of a load, two
// barriers and the products, about 1.5 us: with eight steps at least, small shells ran on a few blocks, 12 - 16 us a
// shell of 16^3 to 32^3 against 4 - 7 us (Bk Fisher of 32^3 295 -> 255 us, 48^3 529 -> 450, 64^3 685 -> 617 us; two
// steps at least 263, 462 and 619 us; from 96^3 on all the same).
static int shell_parts(int64_t n_modes, int n_cols, int64_t *per_block) {
    const int64_t steps = std::max<int64_t>(1, (n_modes + SR_M - 1) / SR_M), tiles = (n_cols + SR_CT - 1) / SR_CT;
    const int64_t parts = std::max<int64_t>(1, std::min<int64_t>((3LL * num_sms() + tiles - 1) / tiles, steps));
    *per_block = (steps + parts - 1) / parts * SR_M;
    return (int)std::max<int64_t>(1, (n_modes + *per_block - 1) / *per_block);
}

struct ShellRowOut {
    int32_t orow[SR_R];
};

__global__ void shell_rows_finalize(const double *partials, int n_chunks, int n_rows, int n_cols, double scale,
                                    double *out, int64_t out_stride, ShellRowOut o) {
    const int t = blockIdx.x * SUM_COLS + threadIdx.x;
    const int total = n_rows * n_cols;
    const double s = block_column_sum(partials + t, total, n_chunks, t < total);
    if (threadIdx.y != 0 || t >= total) return;
    const int r = t / n_cols, j = t - r * n_cols;
    out[(int64_t)o.orow[r] * out_stride + j] = s * scale;
}
}  // namespace pb

extern "C" int pb_shell_rows_workspace_size(int64_t n_modes, int n_rows, int n_cols, size_t *bytes) {
    if (!bytes) return fail(PB_ERR_INVALID, "bytes is NULL");
    if (n_modes < 0 || n_rows < 1 || n_rows > SR_R || n_cols < 1)
        return fail(PB_ERR_INVALID, "pb_shell_rows_workspace_size: bad sizes");
    int64_t per_block;
    *bytes = (size_t)shell_parts(n_modes, n_cols, &per_block) * n_rows * n_cols * sizeof(double);
    return PB_OK;
}

extern "C" int pb_shell_rows(const pb_grid_t *g, int precision, const void *F, int n_f, const void *Q, int n_cols,
                             const int64_t *modes, int64_t n_modes, const int32_t *row_key, const int32_t *out_row,
                             int n_rows, double scale, double *out, int64_t out_stride, void *workspace,
                             size_t workspace_bytes, void *stream) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!F || !Q || !row_key || !out_row || !out) return fail(PB_ERR_INVALID, "pb_shell_rows: NULL argument");
    if (n_rows < 1 || n_rows > SR_R) return fail(PB_ERR_INVALID, "pb_shell_rows: n_rows must be in [1, 32]");
    if (n_cols < 1 || n_f < 1) return fail(PB_ERR_INVALID, "pb_shell_rows: empty input");
    if (n_modes < 0 || (n_modes > 0 && !modes)) return fail(PB_ERR_INVALID, "pb_shell_rows: bad mode list");
    ShellRowKeys keys;
    ShellRowOut orow;
    for (int r = 0; r < SR_R; ++r) {
        keys.key[r] = r < n_rows ? row_key[r] : 0;
        orow.orow[r] = r < n_rows ? out_row[r] : 0;
        if (r < n_rows && (keys.key[r] < 0 || keys.key[r] >= n_f))
            return fail(PB_ERR_INVALID, "pb_shell_rows: row key out of range");
        if (r < n_rows && orow.orow[r] < 0) return fail(PB_ERR_INVALID, "pb_shell_rows: negative output row");
    }
    if (out_stride == 0) out_stride = n_cols;
    int64_t per_block;
    const int n_chunks = shell_parts(n_modes, n_cols, &per_block);  // an empty shell: one block of zeros
    size_t need = (size_t)n_chunks * n_rows * n_cols * sizeof(double);
    if (!workspace || workspace_bytes < need) return fail(PB_ERR_WORKSPACE, "pb_shell_rows: workspace too small");
    cudaStream_t s = as_stream(stream);
    dim3 grid((unsigned)n_chunks, (n_cols + SR_CT - 1) / SR_CT);
    double *partials = (double *)workspace;
    if (precision != PB_F64 && precision != PB_F32) return fail(PB_ERR_INVALID, "bad precision");
#define PB_SR_LAUNCH(T, RPT)                                                                                       \
    shell_rows_kernel<T, RPT><<<grid, SR_THREADS, 0, s>>>(G, (const cplx<T>::type *)F, (const cplx<T>::type *)Q,   \
                                                          n_rows, n_cols, modes, n_modes, per_block, keys, partials)
#define PB_SR_ROWS(T)                              \
    switch ((n_rows + 7) / 8) {                    \
        case 1: PB_SR_LAUNCH(T, 1); break;         \
        case 2: PB_SR_LAUNCH(T, 2); break;         \
        case 3: PB_SR_LAUNCH(T, 3); break;         \
        default: PB_SR_LAUNCH(T, 4); break;        \
    }
    if (precision == PB_F64) PB_SR_ROWS(double)
    else PB_SR_ROWS(float)
#undef PB_SR_ROWS
#undef PB_SR_LAUNCH
    PB_LAUNCH_CHECK("pb_shell_rows");
    int total = n_rows * n_cols;
    shell_rows_finalize<<<(total + SUM_COLS - 1) / SUM_COLS, dim3(SUM_COLS, SUM_ROWS), 0, s>>>(
        partials, (int)n_chunks, n_rows, n_cols, scale, out, out_stride, orow);
    PB_LAUNCH_CHECK("pb_shell_rows(finalize)");
    return PB_OK;
}

// ------------------------------------------------------------------------------------
// pb_bin_reduce_noalloc: the k-bin reduction with its scratch in a fixed device array.
//
// Some callers cannot hand this library a workspace: a binding that only forwards the
// input and output pointers it was given and owns no device allocator, or a host program
// whose GPU memory is entirely reserved by another framework's pool, where a cudaMalloc
// (which may also synchronise the device) is not acceptable.  For them the per-block
// partial sums live in the file-scope array below, PB_BIN_REDUCE_NOALLOC_MAX_DOUBLES
// doubles (2 MiB); every GPU that loads the library keeps it until the process exits.
//
// The array's host-side name is only a stand-in for the device symbol, so its device
// address is looked up once per device with cudaGetSymbolAddress, with that device
// current, on the first call made on that device; make that first call before any stream
// capture.  The address is kept for the life of the process: a program that resets the
// device (cudaDeviceReset) must not call this entry point afterwards.  All calls share the
// one array: calls whose kernels overlap on the GPU (other streams, other host threads)
// race on it and must be serialised by the caller.  Each call writes every partial it later
// reads, so nothing is carried over from the previous call.  Spectra go through the same
// deterministic multi-row kernel as pb_bin_reduce, with as many blocks per row as fit.
// ------------------------------------------------------------------------------------
#include <mutex>

namespace pb {
static __device__ __align__(256) double g_binred_scratch[PB_BIN_REDUCE_NOALLOC_MAX_DOUBLES];

static std::mutex g_binred_scratch_mu;
static double *g_binred_scratch_dev[64];  // device address per device ordinal, looked up once

static int binred_scratch_address(double **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_check(e, "pb_bin_reduce_noalloc: cudaGetDevice");
    if (dev < 0 || dev >= 64) return fail(PB_ERR_UNSUPPORTED, "pb_bin_reduce_noalloc: device ordinal >= 64");
    std::lock_guard<std::mutex> lock(g_binred_scratch_mu);
    if (!g_binred_scratch_dev[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_binred_scratch);
        if (e != cudaSuccess) return cuda_check(e, "pb_bin_reduce_noalloc: cudaGetSymbolAddress");
        g_binred_scratch_dev[dev] = (double *)p;
    }
    *out = g_binred_scratch_dev[dev];
    return PB_OK;
}
}  // namespace pb

extern "C" int pb_bin_reduce_noalloc(const pb_grid_t *g, int precision, int mode, const void *a, const void *b,
                                     int n_rows, int64_t row_stride, const double *edges, int nk,
                                     const int32_t *ells, int n_ell, double scale, double *out, int accumulate,
                                     void *stream) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (nk < 1 || nk > PB_RED_MAX_BINS) return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: nk must be in [1, 64]");
    if (n_ell < 1 || n_ell > PB_RED_MAX_ELLS)
        return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: n_ell must be in [1, 9]");
    if (n_rows < 1 || n_rows > 65535)
        return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: n_rows must be in [1, 65535]");
    if (!edges || !ells || !out) return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: NULL argument");
    if (mode == PB_RED_ABS2 && !a) return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: ABS2 needs a");
    if (mode == PB_RED_CROSS && (!a || !b)) return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: CROSS needs a and b");
    if (mode < 0 || mode > 2) return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: bad mode");
    if (precision != PB_F32 && precision != PB_F64) return fail(PB_ERR_INVALID, "bad precision");
    // partial sums: one slot of n_ell*nk doubles per (row, block); shrink the block count
    // to fit the fixed array, down to one block per row
    const int64_t per_row_block = (int64_t)nk * n_ell;
    const int64_t fit = PB_BIN_REDUCE_NOALLOC_MAX_DOUBLES / ((int64_t)n_rows * per_row_block);
    if (fit < 1)
        return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: n_rows * nk * n_ell = " +
                                        std::to_string((int64_t)n_rows * per_row_block) +
                                        " doubles exceeds the fixed scratch of " +
                                        std::to_string((int64_t)PB_BIN_REDUCE_NOALLOC_MAX_DOUBLES) +
                                        "; use pb_bin_reduce with a workspace");
    if (row_stride == 0) row_stride = G.nhalf;
    RedParams p;
    for (int i = 0; i <= nk; ++i) {
        p.edges[i] = edges[i];
        if (i > 0 && !(edges[i] > edges[i - 1]))
            return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: bin edges must be strictly increasing");
    }
    for (int e = 0; e < n_ell; ++e) {
        if (ells[2 * e] < 0 || ells[2 * e] > 4 || ells[2 * e + 1] < 0 || ells[2 * e + 1] > 4)
            return fail(PB_ERR_INVALID, "pb_bin_reduce_noalloc: Legendre order must be in [0, 4]");
        p.la[e] = (int8_t)ells[2 * e];
        p.lb[e] = (int8_t)ells[2 * e + 1];
    }
    p.nk = nk;
    p.n_ell = n_ell;
    double *partials = nullptr;
    st = binred_scratch_address(&partials);
    if (st) return st;
    int nb = (int)std::min<int64_t>(red_blocks(G), fit);
    cudaStream_t s = as_stream(stream);
    if (mode != PB_RED_REAL2) {
        // spectra: the deterministic multi-row kernel of pb_bin_reduce (its accumulators are
        // dynamic shared memory, not device memory), on the block count that fits the array
        const int per = nk * n_ell;
        const int rpg = std::max(1, std::min(n_rows, RR_ACC_DOUBLES / per));
        const size_t smem = rr_acc_len(rpg, n_ell, nk) * sizeof(double) + (size_t)n_ell * RR_TILE * sizeof(double) +
                            (size_t)RR_TILE * (sizeof(double2) + sizeof(int));
        dim3 rgrid(nb, (n_rows + rpg - 1) / rpg);
#define PB_RR_LAUNCH(T, M)                                                                                   \
    do {                                                                                                     \
        PB_CUDA(cudaFuncSetAttribute(binred_rows_kernel<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)smem));                                                            \
        binred_rows_kernel<T, M><<<rgrid, RED_THREADS, smem, s>>>(G, (const cplx<T>::type *)a,              \
                                                                  (const cplx<T>::type *)b, row_stride, p,   \
                                                                  n_rows, rpg, partials);                    \
    } while (0)
        if (precision == PB_F32) {
            if (mode == PB_RED_ABS2) PB_RR_LAUNCH(float, PB_RED_ABS2);
            else PB_RR_LAUNCH(float, PB_RED_CROSS);
        } else {
            if (mode == PB_RED_ABS2) PB_RR_LAUNCH(double, PB_RED_ABS2);
            else PB_RR_LAUNCH(double, PB_RED_CROSS);
        }
#undef PB_RR_LAUNCH
    } else {
        dim3 grid(nb, n_rows);
        if (precision == PB_F32)
            binred_kernel<float, PB_RED_REAL2><<<grid, RED_THREADS, 0, s>>>(G, nullptr, nullptr, (const float *)a,
                                                                            row_stride, p, partials);
        else
            binred_kernel<double, PB_RED_REAL2><<<grid, RED_THREADS, 0, s>>>(G, nullptr, nullptr, (const double *)a,
                                                                             row_stride, p, partials);
    }
    PB_LAUNCH_CHECK("pb_bin_reduce_noalloc");
    launch_binred_finalize(partials, nb, nk * n_ell, n_rows, scale, out, accumulate, s);
    PB_LAUNCH_CHECK("pb_bin_reduce_noalloc(finalize)");
    return PB_OK;
}
