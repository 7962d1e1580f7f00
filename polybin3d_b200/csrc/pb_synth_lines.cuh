// Band-limited map synthesis on pb_fft.cuh (pb_shell_synth, plain maps):
//   out[m](x) = sum_k F_m(k) e^{+2 pi i k.x / M},
//   F_m(k)    = scale_m src[src_m](k) w(k)^wpow_m Theta(lo_m <= |k| < hi_m) L_l1(mu) L_l2(mu)
// in three passes over W[map][x][y][kz] (kz <= the maps' band, rows of whole 128-byte lines):
//   X  per (map, ky in the band, run of kz): gather + filter + inverse transform along x
//   Y  per (map, x, run of kz): inverse transform along y, in place
//   Z  per (map, pairs of rows (x, y), (x, y + 1)): two Hermitian rows packed into one complex line,
//      inverse transform along z, two real rows out
// Every global access is a run along kz or z of at least 64 bytes (the passes before read and wrote
// [kz][x][y] planes, with kz outermost), an exchange between passes is all that goes through shared memory (one
// for most lengths up to 256), and the operands of a thread's 8 - 16-point butterfly are in flight together.
// Measured on a B200, 32 FP32 maps on 192^3 from a 256^3 spectrum (the bispectrum of 16 bins, l = 0,
// 2): 637 us against 763 us for 32 FP32 maps on 192^3, 215 against 664 us for 24 FP64 maps on 120^3.
#pragma once
#include <cuda_bf16.h>
#include "pb_fft.cuh"

namespace pb {

constexpr int SL_MAX_MAPS = 64;

struct SlMap {
    double lo, hi;         // thresholds on |k|^2
    double lo2, hi2;       // squares of the edges (index ranges)
    double scale;
    int64_t w_off;         // first element of the map's W, rows of ldz
    int32_t src, kz_max, ldz;
    int8_t l1, l2, wpow, pad;
};
struct SlParams {
    Grid g;                          // source grid (frequencies, line of sight)
    int m0, m1, m2, kz_top;          // output grid, largest kz of any map
    int64_t src_stride;
    fft::Axis ax, ay, az;
    int tab_y, tab_z;                // offsets of the axes' twiddles in the table
    int t_maps, t_factor;            // a tiled set's map and factor-map counts (0: plain maps)
    SlMap maps[SL_MAX_MAPS];
};

template <typename T> struct SlShape;
// lines of 16 (FP64) or 32 (FP32) kz: 256 bytes
template <> struct SlShape<double> { static constexpr int LINES = 16, THREADS = 128, BLOCKS = 5, ZBLOCKS = 4, ANY = 3; };
template <> struct SlShape<float> { static constexpr int LINES = 32, THREADS = 256, BLOCKS = 3, ZBLOCKS = 8, ANY = 5; };
constexpr int SL_SMEM = 100 * 1024;

template <typename T> __host__ __device__ constexpr size_t sl_line_bytes(const fft::Axis &ax, int L) {
    return ((size_t)ax.tw_len + (size_t)(ax.np - 1) * L * ax.n) * 2 * sizeof(T);
}
template <typename T> __host__ __device__ constexpr int sl_lines(const fft::Axis &ax) {
    int L = SlShape<T>::LINES;
    while (L > 2 && sl_line_bytes<T>(ax, L) > (size_t)SL_SMEM) L /= 2;
    // three passes (two exchange buffers): four blocks per SM, down to runs of 64 bytes (16 FP32 maps of 320^3 2.54 ms with
    // the larger blocks, 2.33 so; runs of 32 bytes at 480 points 8.0 against 7.4 ms)
    while (ax.np == 3 && L * 2 * sizeof(T) > 64 && sl_line_bytes<T>(ax, L) > (size_t)54 * 1024) L /= 2;
    return L;
}
// threads per line: equal rounds of butterflies in the first pass
template <typename T> __host__ __device__ constexpr int sl_threads(const fft::Axis &ax) {
    const int most = SlShape<T>::THREADS / sl_lines<T>(ax), rounds = (ax.nb[0] + most - 1) / most;
    return (ax.nb[0] + rounds - 1) / rounds;
}
// threads per line of the z pass: eight for two passes (16 for 192 took 386 against 348 us for 32 FP32 maps: a
// quarter of them idle in the first pass), the count from 16 to 32 with the fewest idle butterfly slots for three (eight,
// with no idle slot, left 384 points four blocks of 64 threads per SM: 16 FP64 maps of 384^3 10.2 ms, with 32 threads a
// line 6.3 ms)
__host__ __device__ constexpr int sl_z_threads(const fft::Axis &ax) {
    int best = 1, cost = 1 << 30;
    for (int t = ax.np == 1 ? 1 : ax.np == 2 ? 8 : 16; t <= (ax.np == 3 ? 32 : 8); ++t) {
        int c = 0;
        for (int q = 0; q < ax.np; ++q) c += (ax.nb[q] + t - 1) / t * t * ax.R[q];
        if (c <= cost) {
            cost = c;
            best = t;
        }
    }
    return best;
}
template <typename T> __host__ __device__ constexpr size_t sl_z_bytes(const fft::Axis &ax, int pairs) {
    return ((size_t)ax.tw_len + (size_t)(ax.np == 3 ? 2 : 1) * pairs * fft::row_len(ax)) * 2 * sizeof(T);
}
template <typename T> __host__ __device__ constexpr int sl_z_pairs(const fft::Axis &ax) {
    int L = 128 / sl_z_threads(ax);
    if (L < 1) L = 1;
    while (L > 1 && sl_z_bytes<T>(ax, L) > (size_t)SL_SMEM) L /= 2;
    return L;
}

// largest index that may hold modes below the radius (one of margin), -1: none; ky at runs of 32 kz
__device__ __forceinline__ int sl_radius(double r2, double d2, double kf) {
    return d2 < r2 ? (int)(sqrt(r2 - d2) / kf) + 1 : -1;
}
__device__ __forceinline__ int sl_ky_radius(const Grid &g, double r2, int kz) {
    const double z = (kz & ~31) * g.kf2;
    return sl_radius(r2, z * z, g.kf1);
}
template <typename V> __device__ __forceinline__ V &sl_elem(V *p, int e, int stride_bytes) {
    return *reinterpret_cast<V *>(reinterpret_cast<char *>(const_cast<typename std::remove_const<V>::type *>(p)) +
                                  (int64_t)e * stride_bytes);
}

template <typename T> __device__ __forceinline__ void sl_twiddles(const fft::Axis &ax, typename cplx<T>::type *tw, int t, int nt) {
    for (int q = 1; q < ax.np; ++q) {
        const int ns = ax.ns[q], cnt = (ax.R[q] - 1) * ns;
        for (int i = t; i < cnt; i += nt) {
            const int r = i / ns + 1, jm = i - (r - 1) * ns;
            double s, c;
            sincospi(2.0 * (r * jm) / (double)(ns * ax.R[q]), &s, &c);
            typename cplx<T>::type v;
            v.x = (T)c;
            v.y = (T)s;
            tw[ax.tw[q] + i] = v;
        }
    }
}
template <typename C> __device__ __forceinline__ void sl_load_table(C *dst, const C *src, int n) {
    for (int i = threadIdx.y * blockDim.x + threadIdx.x; i < n; i += blockDim.x * blockDim.y) dst[i] = src[i];
}

// ---- X: filter + inverse transform along x ---------------------------------------------
// block (lines of kz, threads per line); grid (source columns ky x runs, maps).  The first block also
// writes the other passes' twiddles.  S: the source's element type (FP32 maps may come from an FP64 spectrum:
// the filter product is formed in FP64 and rounded once)
template <typename T, typename S, int N>
__global__ void __launch_bounds__(SlShape<T>::THREADS, SlShape<T>::BLOCKS)
    sl_x_kernel(const __grid_constant__ SlParams p, const S *src, const T *w, typename cplx<T>::type *table,
                typename cplx<T>::type *W) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const Grid &g = p.g;
    const SlMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.ax);
    const fft::Axis &ax = use.v;
    // one butterfly per thread: the count is hidden from the compiler, which without the loop around it
    // keeps the filters of all its elements at once and spills 700 to 800 bytes a thread (24 FP32 maps from FP64: on 64^3
    // 51 us, 13 with the loop, on 128^3 124 and 42; lengths of two rounds lose 4 % to the hidden count)
    const int L = N ? sl_lines<T>(ax) : blockDim.x, NT = N && sl_threads<T>(ax) < ax.nb[0] ? sl_threads<T>(ax) : blockDim.y,
              runs = p.kz_top / L + 1;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0 && blockIdx.y == 0) {
        sl_twiddles<T>(p.ay, table + p.tab_y, tid, blockDim.x * blockDim.y);
        sl_twiddles<T>(p.az, table + p.tab_z, tid, blockDim.x * blockDim.y);
    }
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, p.m1);                  // the band lies inside both grids
    if (kz0 > mp.kz_max || abs(ky) > sl_ky_radius(g, mp.hi2, kz0)) return;
    C *tw = reinterpret_cast<C *>(sl_smem), *sm = tw + ax.tw_len, *sm2 = sm + ax.n * L;
    sl_twiddles<T>(ax, tw, tid, blockDim.x * blockDim.y);
    const int line = threadIdx.x, kz = kz0 + line;
    const bool on = kz <= mp.kz_max;
    const double kyv = __dmul_rn((double)ky, g.kf1), kzv = __dmul_rn((double)kz, g.kf2);
    const double ky2 = __dmul_rn(kyv, kyv), kz2 = __dmul_rn(kzv, kzv);
    const int r_out = sl_radius(mp.hi2, ky2 + kz2, g.kf0), r_in = sl_radius(mp.lo2, ky2 + kz2, g.kf0) - 2;
    const int64_t col = (int64_t)(ky < 0 ? ky + g.n1 : ky) * g.nh2 + kz, xstep = (int64_t)g.n1 * g.nh2;
    const S *s0 = src ? src + mp.src * p.src_stride + col : nullptr;   // NULL: unit spectrum
    const int wx = p.m1 * mp.ldz * (int)sizeof(C);
    C *o = W + mp.w_off + (int64_t)iy * mp.ldz + kz;
    fft::line_fft<T, 1>(
        use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int e, int side) {
            C v;
            v.x = v.y = (T)0;
            const int ka = fft::abs_label(e, ax.n, side);
            if (ka > r_out || ka < r_in) return v;
            const int kx = (side ? side > 0 : e >= (ax.n >> 1)) ? -ka : ka;
            const double kxv = __dmul_rn((double)kx, g.kf0);
            const double s = __dadd_rn(__dadd_rn(__dmul_rn(kxv, kxv), ky2), kz2);
            if (!(mp.lo <= s && s < mp.hi)) return v;
            const int64_t at = (kx < 0 ? kx + g.n0 : kx) * xstep;
            double f = mp.scale;
            if (mp.l1 | mp.l2) {
                const double k = __dsqrt_rn(s);
                if (mp.l1 > 4) {
                    f *= real_harmonic(mp.l1, kxv, kyv, kzv, k);
                } else {
                    const double mu = k != 0.0 ? __ddiv_rn(k_dot_los(g.los, g.l0, g.l1, g.l2, kxv, kyv, kzv), k) : 0.0;
                    f *= legendre(mp.l1, mu) * legendre(mp.l2, mu);
                }
            }
            if (mp.wpow != 0) {
                const double wv = (double)w[col + at];
                if (mp.wpow == 1) f *= wv;
                else if (mp.wpow == 2) f *= wv * wv;
                else f = wv != 0.0 ? f / wv : 0.0;
            }
            if (s0) {
                const S x = s0[at];
                v.x = (T)((double)x.x * f);
                v.y = (T)((double)x.y * f);
            } else {
                v.x = (T)f;
            }
            return v;
        },
        [&](int x, C v, int) { sl_elem(o, x, wx) = v; });
}

// ---- Y: inverse transform along y, in place ----------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(SlShape<T>::THREADS, SlShape<T>::BLOCKS)
    sl_y_kernel(const __grid_constant__ SlParams p, const typename cplx<T>::type *table, typename cplx<T>::type *W) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const SlMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.ay);
    const fft::Axis &ay = use.v;
    const int L = N ? sl_lines<T>(ay) : blockDim.x, NT = N ? sl_threads<T>(ay) : blockDim.y, runs = p.kz_top / L + 1;
    const int run = blockIdx.x % runs, x = blockIdx.x / runs, kz0 = run * L;
    if (kz0 > mp.kz_max) return;
    C *tw = reinterpret_cast<C *>(sl_smem), *sm = tw + ay.tw_len, *sm2 = sm + ay.n * L;
    sl_load_table(tw, table + p.tab_y, ay.tw_len);
    const int line = threadIdx.x, kz = kz0 + line, row = mp.ldz * (int)sizeof(C);
    const bool on = kz <= mp.kz_max;
    const int ry = sl_ky_radius(p.g, mp.hi2, kz);
    C *w = W + mp.w_off + (int64_t)x * p.m1 * mp.ldz + kz;
    fft::line_fft<T, 1>(
        use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int e, int side) {
            C v;
            v.x = v.y = (T)0;
            if (fft::abs_label(e, ay.n, side) <= ry) v = sl_elem(w, e, row);
            return v;
        },
        [&](int y, C v, int) {
            if (kz == 0) v.y = (T)0;  // the z pass reads the real part of the plane kz = 0
            sl_elem(w, y, row) = v;
        });
}

// ---- Z: two rows per complex line, real rows out ------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(128, SlShape<T>::ZBLOCKS)
    sl_z_kernel(const __grid_constant__ SlParams p, const typename cplx<T>::type *table, const typename cplx<T>::type *W,
                T *out) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const SlMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.az);
    const fft::Axis &az = use.v;
    const int nt = N ? sl_z_threads(az) : blockDim.x, L = N ? sl_z_pairs<T>(az) : blockDim.y, n = az.n, ld = fft::row_len(az);
    C *tw = reinterpret_cast<C *>(sl_smem), *sm = tw + az.tw_len + threadIdx.y * ld, *sm2 = sm + L * ld;
    sl_load_table(tw, table + p.tab_z, az.tw_len);
    const int64_t pair = (int64_t)blockIdx.x * L + threadIdx.y, pairs = (int64_t)p.m0 * p.m1 / 2;
    const bool on = pair < pairs;
    const C *wa = W + mp.w_off + (on ? 2 * pair * mp.ldz : 0), *wb = wa + mp.ldz;
    T *oa = out + ((int64_t)blockIdx.y * pairs + (on ? pair : 0)) * 2 * n, *ob = oa + n;
    const int K = mp.kz_max;
    fft::line_fft<T, 1>(
        use, threadIdx.x, nt, on, sm, sm2, tw, [&](int e) { return fft::row_at(az, e); },
        [&](int e, int side) {
            const bool up = side ? side > 0 : 2 * e > n;
            const int kz = up ? n - e : e;
            C v;
            v.x = v.y = (T)0;
            if (kz > K) return v;
            const C a = wa[kz], b = wb[kz];
            v.x = up ? a.x + b.y : a.x - b.y;
            v.y = up ? b.x - a.y : a.y + b.x;
            return v;
        },
        [&](int z, C v, int) {
            oa[z] = v.x;
            ob[z] = v.y;
        });
}

// ---- tiled-set output ------------------------------------------------------------------
// voxel v of map m into a tiled set: FP32 copy of a factor map, bf16 hi and lo parts
__device__ __forceinline__ void tiled_put(int t_maps, int t_factor, int m, int64_t v, float val, char *out) {
    if (m < t_factor) *reinterpret_cast<float *>(out + tiled_factor_byte(v, m, t_maps, t_factor)) = val;
    const __nv_bfloat16 hi = __float2bfloat16_rn(val);
    const __nv_bfloat16 lo = __float2bfloat16_rn(val - __bfloat162float(hi));
    *reinterpret_cast<__nv_bfloat16 *>(out + tiled_c_byte(v, m, t_maps, t_factor)) = hi;
    *reinterpret_cast<__nv_bfloat16 *>(out + tiled_c_byte(v, tiled_cpad(t_maps) + m, t_maps, t_factor)) = lo;
}

// Staged values of map m (rows of NN voxels, row stride lds in stg; voxels v0 .. v0 + rows NN
// - 1) into a tiled set, by warps wk = 0 .. nw - 1 of a group (the caller's warp index in it).
// Each warp takes 64 consecutive voxels per step, a lane two neighbours: two 128-byte rows of
// factor slabs (8-byte stores) and four 32-byte K-step rows each of the hi and lo parts
// (bf16x2 stores), so the stores fill whole sectors; offsets inside a tile are per lane and
// computed once per map, the tile base per chunk.  Per voxel (tiled_put) when the run is not
// 64-aligned.
__device__ __forceinline__ void flush_tiled(int t_maps, int t_factor, int m, int64_t v0, int rows, int NN, int lds,
                                            const float *stg, char *out, int wk, int nw) {
    const int count = rows * NN;
    const int lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31;
    if ((NN & 1) != 0 || (v0 & 63) != 0 || (count & 63) != 0) {
        for (int i = wk * 32 + lane; i < count; i += nw * 32) {
            const int r = i / NN, z = i - r * NN;
            tiled_put(t_maps, t_factor, m, v0 + i, stg[r * lds + z], out);
        }
        return;
    }
    const int F = tiled_frows(t_factor), P = tiled_cpad(t_maps);
    const int64_t tb = tiled_tile_bytes(t_maps, t_factor);
    const bool factor = m < t_factor;
    // lane j holds voxels 2j, 2j + 1 of the chunk: slab j / 16, 4-voxel chunk (j % 16) / 2 of
    // it; K step j / 8, 8-voxel half (j / 4) % 2, element 2 (j % 4)
    const uint32_t off_f = (uint32_t)(lane >> 4) * F * 128u + (uint32_t)m * 128u +
                           ((((uint32_t)(lane & 15) >> 1) ^ ((uint32_t)m & 7u)) << 4) + (lane & 1) * 8;
    auto c_off = [&](int r) {
        return (uint32_t)((lane >> 3) * 64 * P + (r >> 3) * 256 + (r & 7) * 32 +
                          ((((lane >> 2) & 1) ^ ((r >> 2) & 1)) << 4) + (lane & 3) * 4);
    };
    const uint32_t off_hi = c_off(m), off_lo = c_off(P + m);
    for (int u = wk * 64; u < count; u += nw * 64) {
        const int i = u + 2 * lane, r = i / NN, z = i - r * NN;  // NN even: both voxels in row r
        const float x0 = stg[r * lds + z], x1 = stg[r * lds + z + 1];
        const int64_t v = v0 + u;  // 64-aligned: two slabs, four K steps of one tile
        const int w = (int)(v & (TILED_VOX - 1));
        char *const tile = out + (v >> 7) * tb;
        if (factor) *reinterpret_cast<float2 *>(tile + (w >> 5) * F * 128 + off_f) = make_float2(x0, x1);
        const __nv_bfloat162 hb = __floats2bfloat162_rn(x0, x1);
        const __nv_bfloat162 lb = __floats2bfloat162_rn(x0 - __low2float(hb), x1 - __high2float(hb));
        char *const cop = tile + 512 * F + (w >> 4) * 64 * P;
        *reinterpret_cast<__nv_bfloat162 *>(cop + off_hi) = hb;
        *reinterpret_cast<__nv_bfloat162 *>(cop + off_lo) = lb;
    }
}

// ---- Z into a tiled set: a block per (pairs of rows, group of SL_TMAPS maps) ----------------
// Its lines are (map, pair) combinations, so the block writes neighbouring maps' rows of the same tiles --
// one 8-row atom of each factor slab and K step -- together; rows are staged in shared memory
// and flushed in whole sectors.  Same arithmetic as sl_z_kernel: factor rows equal the plain maps.
constexpr int SL_TMAPS = 8;
__host__ __device__ constexpr size_t sl_tile_bytes(const fft::Axis &az, int pairs) {
    const int L = SL_TMAPS * pairs;
    return sl_z_bytes<float>(az, L) + (size_t)2 * L * (az.n + 1) * sizeof(float);
}
__host__ __device__ constexpr int sl_tile_pairs(const fft::Axis &az) {
    return sl_z_threads(az) <= 16 && sl_tile_bytes(az, 2) <= (size_t)110 * 1024 ? 2 : 1;
}
template <int N>
__global__ void __launch_bounds__(256, 2)
    sl_z_tiled_kernel(const __grid_constant__ SlParams p, const float2 *table, const float2 *W, int n_maps, char *out) {
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const fft::AxisUse<N, true> use(p.az);
    const fft::Axis &az = use.v;
    const int nt = N ? sl_z_threads(az) : blockDim.x, LY = N ? sl_tile_pairs(az) : blockDim.y / SL_TMAPS, L = SL_TMAPS * LY, n = az.n,
              ld = fft::row_len(az), lds = n + 1;
    float2 *tw = reinterpret_cast<float2 *>(sl_smem), *buf = tw + az.tw_len;
    float *stg = reinterpret_cast<float *>(buf + (size_t)(az.np == 3 ? 2 : 1) * L * ld);
    float2 *sm = buf + threadIdx.y * ld, *sm2 = sm + L * ld;
    sl_load_table(tw, table + p.tab_z, az.tw_len);
    const int line = threadIdx.y, mi = line / LY, m0 = blockIdx.y * SL_TMAPS, nm = min(SL_TMAPS, n_maps - m0);
    const int64_t pairs = (int64_t)p.m0 * p.m1 / 2, q0 = (int64_t)blockIdx.x * LY, pair = q0 + line - mi * LY;
    const bool on = mi < nm && pair < pairs;
    const SlMap &mp = p.maps[on ? m0 + mi : 0];
    const float2 *wa = W + mp.w_off + (on ? 2 * pair * mp.ldz : 0), *wb = wa + mp.ldz;
    const int K = mp.kz_max;
    fft::line_fft<float, 1>(
        use, threadIdx.x, nt, on, sm, sm2, tw, [&](int e) { return fft::row_at(az, e); },
        [&](int e, int side) {
            const bool up = side ? side > 0 : 2 * e > n;
            const int kz = up ? n - e : e;
            if (kz > K) return make_float2(0.f, 0.f);
            const float2 a = wa[kz], b = wb[kz];
            return up ? make_float2(a.x + b.y, b.x - a.y) : make_float2(a.x - b.y, a.y + b.x);
        },
        [&](int z, float2 v, int) {
            stg[(2 * line) * lds + z] = v.x;
            stg[(2 * line + 1) * lds + z] = v.y;
        });
    __syncthreads();
    const int rows = 2 * (int)min((int64_t)LY, pairs - q0);
    // a warp handles whole maps in turn (the block's size need not be a multiple of 32)
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, nw = blockDim.x * blockDim.y / 32, warp = tid >> 5;
    if (nw == 0) {
        for (int k = 0; k < nm; ++k)
            for (int i = tid; i < rows * n; i += blockDim.x * blockDim.y) {
                const int r = i / n;
                tiled_put(p.t_maps, p.t_factor, m0 + k, 2 * q0 * n + i, stg[(2 * k * LY + r) * lds + i - r * n], out);
            }
    } else if (warp < nw)
        for (int k = warp; k < nm; k += nw)
            flush_tiled(p.t_maps, p.t_factor, m0 + k, 2 * q0 * n, rows, n, lds, stg + 2 * k * LY * lds, out, 0, 1);
}

// ---- launches -------------------------------------------------------------------------------
enum SlStage { SL_X, SL_Y, SL_Z, SL_Z_TILED };
struct SlArgs {
    const void *src, *w;
    void *table, *W, *out;
    int n_maps;
};

template <typename K> static cudaError_t sl_allow(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <typename T, typename S, int N> cudaError_t sl_launch_x(const SlParams &p, const SlArgs &a, cudaStream_t s) {
    using C = typename cplx<T>::type;
    const int L = sl_lines<T>(p.ax), t = sl_threads<T>(p.ax), runs = p.kz_top / L + 1;
    const size_t smem = sl_line_bytes<T>(p.ax, L);
    const cudaError_t e = sl_allow(sl_x_kernel<T, S, N>, smem);
    if (e != cudaSuccess) return e;
    sl_x_kernel<T, S, N><<<dim3((unsigned)(p.m1 * runs), a.n_maps), dim3(L, t), smem, s>>>(
        p, (const S *)a.src, (const T *)a.w, (C *)a.table, (C *)a.W);
    return cudaGetLastError();
}

// one pass with the kernels of length N (0: the run-time plan)
template <typename T, typename S, int N>
cudaError_t sl_launch(SlStage stage, const SlParams &p, const SlArgs &a, cudaStream_t s) {
    using C = typename cplx<T>::type;
    cudaError_t e;
    if (stage == SL_Z) {
        const int t = sl_z_threads(p.az), L = sl_z_pairs<T>(p.az);
        const size_t smem = sl_z_bytes<T>(p.az, L);
        if ((e = sl_allow(sl_z_kernel<T, N>, smem)) != cudaSuccess) return e;
        const int64_t pairs = (int64_t)p.m0 * p.m1 / 2;
        sl_z_kernel<T, N><<<dim3((unsigned)((pairs + L - 1) / L), a.n_maps), dim3(t, L), smem, s>>>(
            p, (const C *)a.table, (const C *)a.W, (T *)a.out);
        return cudaGetLastError();
    }
    if (stage == SL_Z_TILED) {
        if constexpr (std::is_same<T, float>::value) {
            const int L = SL_TMAPS * sl_tile_pairs(p.az), LY = sl_tile_pairs(p.az);
            const size_t smem = sl_tile_bytes(p.az, LY);
            if ((e = sl_allow(sl_z_tiled_kernel<N>, smem)) != cudaSuccess) return e;
            const int64_t pairs = (int64_t)p.m0 * p.m1 / 2;
            sl_z_tiled_kernel<N><<<dim3((unsigned)((pairs + LY - 1) / LY), (a.n_maps + SL_TMAPS - 1) / SL_TMAPS),
                                   dim3(sl_z_threads(p.az), L), smem, s>>>(p, (const C *)a.table, (const C *)a.W, a.n_maps,
                                                                          (char *)a.out);
            return cudaGetLastError();
        }
        return cudaErrorInvalidValue;
    }
    if (stage == SL_X) return sl_launch_x<T, S, N>(p, a, s);
    const int L = sl_lines<T>(p.ay), t = sl_threads<T>(p.ay), runs = p.kz_top / L + 1;
    const size_t smem = sl_line_bytes<T>(p.ay, L);
    if ((e = sl_allow(sl_y_kernel<T, N>, smem)) != cudaSuccess) return e;
    sl_y_kernel<T, N><<<dim3((unsigned)(p.m0 * runs), a.n_maps), dim3(L, t), smem, s>>>(p, (const C *)a.table, (C *)a.W);
    return cudaGetLastError();
}

// element types of a synthesis: maps and source
enum SlTypes { SL_F64, SL_F32, SL_F32_SRC64 };
template <int N>
cudaError_t sl_dispatch(SlTypes ty, SlStage stage, const SlParams &p, const SlArgs &a, cudaStream_t s) {
    if (ty == SL_F64) return sl_launch<double, double2, N>(stage, p, a, s);
    if (ty == SL_F32 || stage != SL_X) return sl_launch<float, float2, N>(stage, p, a, s);
    return sl_launch<float, double2, N>(stage, p, a, s);
}

// lengths with kernels of their own, as MR_GROUP_* (pb_masked.cuh); the groups spread the compilation
#define SL_GROUP_0(X) X(48) X(60) X(64) X(72) X(80)
#define SL_GROUP_1(X) X(90) X(96) X(100) X(108) X(120)
#define SL_GROUP_2(X) X(128) X(144) X(150) X(160) X(180)
#define SL_GROUP_3(X) X(192) X(200) X(216) X(240) X(256)
#define SL_CASE(N) \
    case N: *e = sl_dispatch<N>(ty, stage, p, a, s); return true;
#define SL_ARGS int n, SlTypes ty, SlStage stage, const SlParams &p, const SlArgs &a, cudaStream_t s, cudaError_t *e
#define SL_DEFINE_GROUP(K)               \
    bool sl_group_##K(SL_ARGS) {         \
        switch (n) { SL_GROUP_##K(SL_CASE) } \
        return false;                    \
    }
// the run-time plan, any other length (a file per type: each takes the compiler a minute or two)
#define SL_ANY_ARGS SlStage stage, const SlParams &p, const SlArgs &a, cudaStream_t s
cudaError_t sl_any_f64(SL_ANY_ARGS);
cudaError_t sl_any_f32(SL_ANY_ARGS);
cudaError_t sl_any_f32_src64(SL_ANY_ARGS);
bool sl_group_0(SL_ARGS);
bool sl_group_1(SL_ARGS);
bool sl_group_2(SL_ARGS);
bool sl_group_3(SL_ARGS);

}  // namespace pb
