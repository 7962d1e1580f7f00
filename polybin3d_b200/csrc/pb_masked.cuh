// Masked rows: Q[m] = rfftn(mask * irfftn(F_m)) for a batch of band-limited half spectra
//   F_m(k) = sum_legs scale * src[s](k) * Theta(lo <= |k| < hi) L_l(mu)
// (the rows of the Monte Carlo Fisher matrices, PolyBin3D/pspec.py:443-456 and
// bspec.py:600-640), FP64, on the modes |k| < k_out that the Fisher sums read.
//
// Filter + batched c2r + mask product + batched r2c moved each map through memory 14 times
// (filter 1, c2r 6, product 2, r2c 6 passes less one) and transformed every line.  Here five passes,
// all of them reading and writing runs of >= 64 contiguous bytes (kz stays the fastest axis):
//   X  per (map, ky, 16 kz): gather + filter + inverse transform along x     src -> W[m][x][ky][kz]
//   Y  per (map, x, 16 kz): inverse transform along y                        W -> W[m][x][y][kz]
//   Z  per (map, pairs of rows (x, y)): two Hermitian rows packed into one complex line, inverse
//      transform along z, times the mask, forward transform, all in registers and shared memory
//   Y' per (map, x, 16 kz): unpack the pairs, forward transform along y      W -> W[m][x][ky][kz]
//   X' per (map, ky, 16 kz): forward transform along x                       W -> Q[m][kx][ky][kz]
// Three kinds of work are never done: columns (ky, kz) outside a map's own band on the way in,
// columns outside k_out on the way out, and rows (x, y) where the mask is zero everywhere (Y
// transforms only planes x that hold such a row, Z only those rows; the rest is exactly zero).
// W holds kz <= k_out / kF only, rows padded to whole 128-byte lines.  X, Y and Z wait for loads (20 warps per SM for the
// x and y passes, 16 for z; 21 - 37 % of the copy rate); memory takes over in the last two passes, Y' 56 % and X' 62 % of
// the copy rate for masked rows, 86 and 79 % for products (32 maps of 128^3).  Chunks of 5 maps whose W stays in L2 took
// longer than chunks of 32 (more blocks per launch, fewer tails).
// Measured on a B200, 60 rows of 128^3 (bins to 0.93 of the Nyquist frequency), against 2.95 ms for
// filter, cuFFT and mask: 0.65 ms on a sector mask (17 % of the rows), 1.23 ms on a ball (71 %).
#pragma once
#include "pb_fft.cuh"

namespace pb {

using fft::Axis;

constexpr int MR_MAX_MAPS = 32;   // maps per chunk
constexpr int MR_MAX_LEGS = 3;
constexpr int MR_THREADS = 256;       // z passes
constexpr int MR_LINE_THREADS = 128;  // x and y passes: five blocks, 20 warps per SM
constexpr int MR_SMEM = 100 * 1024;

struct MrLeg {
    double lo, hi, scale;   // on |k|^2 (exact thresholds), and the factor
    int src, ell;
};
struct MrMap {
    double hi2, lo2;        // squares of the largest upper and smallest lower edge: nothing lies outside
    int kz_max;
    MrLeg leg[MR_MAX_LEGS];
};
struct MrParams {
    Grid g;
    int n_legs, ldz, kz_out;
    double out2;                   // square of k_out (with a margin)
    int64_t src_stride, w_map;     // elements per map of src and W
    int n_x, n_pairs;
    Axis ax, ay, azi, azf;
    int tw_x, tw_y, tw_zi, tw_zf;  // table offsets (complex elements)
    MrMap maps[MR_MAX_MAPS];
};

// lines per block of an x / y transform, and threads per line (one or more equal rounds of
// butterflies in the first pass)
__host__ __device__ constexpr size_t line_bytes(const Axis &ax, int L) {
    return ((size_t)ax.tw_len + (size_t)(ax.np - 1) * L * ax.n) * sizeof(double2);
}
__host__ __device__ constexpr int line_count(const Axis &ax) {
    int L = ax.np == 1 ? 32 : 16;
    while (L > 2 && line_bytes(ax, L) > (size_t)MR_SMEM) L /= 2;
    return L;
}
__host__ __device__ constexpr int line_threads(const Axis &ax) {
    const int most = MR_LINE_THREADS / line_count(ax), rounds = (ax.nb[0] + most - 1) / most;
    return (ax.nb[0] + rounds - 1) / rounds;
}

// Largest index |i| of an axis with fundamental frequency kf for which a column or mode at squared
// distance d2 from it may lie below the radius (one index of margin; the filters test each mode
// exactly); -1: none.  In ky the distance is taken at kz rounded down to a run of 16, whatever the
// lines per block of a pass, so that every pass takes the same columns.
__device__ __forceinline__ int index_radius(double r2, double d2, double kf) {
    return d2 < r2 ? (int)(sqrt(r2 - d2) / kf) + 1 : -1;
}
__device__ __forceinline__ int ky_radius(const Grid &g, double r2, int kz) {
    const double z = (kz & ~15) * g.kf2;
    return index_radius(r2, z * z, g.kf1);
}
// element e of a strided line: one wide multiply-add per address
template <typename T> __device__ __forceinline__ T &elem(T *p, int e, int stride_bytes) {
    return *reinterpret_cast<T *>(reinterpret_cast<char *>(const_cast<typename std::remove_const<T>::type *>(p)) +
                                  (int64_t)e * stride_bytes);
}

__device__ __forceinline__ void load_table(double2 *dst, const double2 *src, int n) {
    const int t = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    for (int i = t; i < n; i += nt) dst[i] = src[i];
}

// ---- X: filter + inverse transform along x ---------------------------------------------
// block (L lines of kz, threads per line); grid (columns x runs, maps)
template <int N>
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_x_kernel(const __grid_constant__ MrParams p, const double2 *src,
                                                            const double2 *table, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.ax);
    const Axis &ax = use.v;
    const int L = N ? line_count(ax) : blockDim.x, NT = N ? line_threads(ax) : blockDim.y, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, g.n1);
    if (kz0 > mp.kz_max || abs(ky) > ky_radius(g, mp.hi2, kz0)) return;
    double2 *tw = mr_smem, *sm = tw + ax.tw_len, *sm2 = sm + ax.n * L;
    load_table(tw, table + p.tw_x, ax.tw_len);
    const int line = threadIdx.x, kz = kz0 + line;
    const bool on = kz <= mp.kz_max;
    const double kyv = __dmul_rn((double)ky, g.kf1), kzv = __dmul_rn((double)kz, g.kf2);
    const double ky2 = __dmul_rn(kyv, kyv), kz2 = __dmul_rn(kzv, kzv);
    // |kx| of the map's shells: only these are tested mode by mode
    const int r_out = index_radius(mp.hi2, ky2 + kz2, g.kf0), r_in = index_radius(mp.lo2, ky2 + kz2, g.kf0) - 2;
    const double2 *s0 = src + (int64_t)iy * g.nh2 + kz;
    const int xs = g.n1 * g.nh2 * (int)sizeof(double2), wx = g.n1 * p.ldz * (int)sizeof(double2);
    double2 *w = W + blockIdx.y * p.w_map + (int64_t)iy * p.ldz + kz;
    fft::line_fft<double, 1>(
        use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int e, int side) {
            double2 v = make_double2(0.0, 0.0);
            const int kx = fft::abs_label(e, ax.n, side);
            if (kx > r_out || kx < r_in) return v;
            const double kxv = __dmul_rn((double)kx, g.kf0);
            const double s = __dadd_rn(__dadd_rn(__dmul_rn(kxv, kxv), ky2), kz2);
            for (int q = 0; q < p.n_legs; ++q) {
                const MrLeg &lg = mp.leg[q];
                if (lg.lo <= s && s < lg.hi) {
                    double f = lg.scale;
                    if (lg.ell) {
                        const double m2 = s > 0.0 ? kz2 / s : 0.0;
                        f *= lg.ell == 2 ? 1.5 * m2 - 0.5 : (35.0 * m2 * m2 - 30.0 * m2 + 3.0) * 0.125;
                    }
                    const double2 x = elem(s0 + lg.src * p.src_stride, e, xs);
                    v.x += f * x.x;
                    v.y += f * x.y;
                }
            }
            return v;
        },
        [&](int x, double2 v, int) { elem(w, x, wx) = v; });
}

// ---- Y: inverse (SIGN 1) and forward (SIGN -1) transforms along y, in place ---------------
// Rows go in pairs (y even, y + 1), the last one alone when n1 is odd; pair_on[x ceil(n1 / 2) + y / 2]:
// the mask is not zero on both (NULL: every pair).  xs: the planes x to do (NULL: all).
template <int SIGN, int N>
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_y_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                            const int32_t *xs, const uint8_t *pair_on, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.ay);
    const Axis &ay = use.v;
    const int L = N ? line_count(ay) : blockDim.x, NT = N ? line_threads(ay) : blockDim.y, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, xi = blockIdx.x / runs, x = xs ? xs[xi] : xi,
              kz0 = run * L;
    const int kz_max = SIGN > 0 ? mp.kz_max : p.kz_out;
    if (kz0 > kz_max) return;
    double2 *tw = mr_smem, *sm = tw + ay.tw_len, *sm2 = sm + ay.n * L;
    load_table(tw, table + p.tw_y, ay.tw_len);
    const int line = threadIdx.x, kz = kz0 + line;
    const bool on = kz <= kz_max;
    __shared__ uint8_t act[512];
    const int half = (g.n1 + 1) / 2;
    for (int i = threadIdx.y * L + line; i < half; i += L * blockDim.y) act[i] = pair_on ? pair_on[x * half + i] : 1;
    __syncthreads();
    double2 *w = W + blockIdx.y * p.w_map + (int64_t)x * g.n1 * p.ldz + kz;
    const int ry = ky_radius(g, SIGN > 0 ? mp.hi2 : p.out2, kz), row = p.ldz * (int)sizeof(double2);
    auto at = [&](int e) { return e * L + line; };
    const double2 zero = make_double2(0.0, 0.0);
    const bool real = kz == 0 || 2 * kz == g.n2;  // planes whose c2r reads real parts only
    if (SIGN > 0) {
        fft::line_fft<double, 1>(
            use, threadIdx.y, NT, on, sm, sm2, tw, at,
            [&](int e, int side) { return fft::abs_label(e, ay.n, side) <= ry ? elem(w, e, row) : zero; },
            [&](int y, double2 v, int) {
                if (real) v.y = 0.0;
                if (act[y >> 1]) elem(w, y, row) = v;
            });
    } else {
        // With F the packed transform of a pair (halved on its way in), row y even holds F[kz] and row
        // y + 1 holds i conj(F[-kz]): the transform of either row is then own - i other.  The other
        // comes from the lane 16 further where that lane reads row y ^ 1 in the same round
        const bool shuffle = L == 16 && (ay.nb[0] & 1) == 0 && (NT & 1) == 0 && (ay.n & 1) == 0;
        const unsigned lanes = __ballot_sync(0xffffffffu, on);
        fft::line_fft<double, -1>(
            use, threadIdx.y, NT, on, sm, sm2, tw, at,
            [&](int y, int) { return act[y >> 1] ? elem(w, y, row) : zero; },
            [&](int e, double2 v, int side) {
                if (fft::abs_label(e, ay.n, side) <= ry) elem(w, e, row) = v;
            },
            [&](int y, double2 v) {
                double2 o;
                if (shuffle) {
                    o.x = __shfl_xor_sync(lanes, v.x, 16);
                    o.y = __shfl_xor_sync(lanes, v.y, 16);
                } else {
                    if ((y ^ 1) >= ay.n) return v;
                    o = act[y >> 1] ? elem(w, y ^ 1, row) : zero;
                }
                return make_double2(v.x + o.y, v.y - o.x);
            });
    }
}

// ---- Z: inverse transform along z, mask, forward transform -------------------------------
// block (threads per line = butterflies of the last inverse pass, L pairs of rows); grid (pairs / L, maps)
template <int N>
__global__ void __launch_bounds__(MR_THREADS, 2) mr_z_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                            const int32_t *pairs, const double *mask, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, false> use_i(p.azi);
    const fft::AxisUse<N, true> use_f(p.azf);
    const Axis &ai = use_i.v, &af = use_f.v;
    const int L = blockDim.y, t = threadIdx.x, nt = N ? ai.nb[ai.np - 1] : blockDim.x, n = ai.n;
    const int ld = max(fft::row_len(ai), fft::row_len(af));
    double2 *twi = mr_smem, *twf = twi + ai.tw_len, *sm = twf + af.tw_len + threadIdx.y * ld;
    double2 *sm2 = sm + L * ld;   // used by three-pass lengths only
    load_table(twi, table + p.tw_zi, ai.tw_len);
    load_table(twf, table + p.tw_zf, af.tw_len);
    const int pr = blockIdx.x * L + threadIdx.y;
    const bool on = pr < p.n_pairs;
    const int ra = on ? pairs[pr] : 0, rb = on && (ra % g.n1) + 1 < g.n1 ? ra + 1 : -1;
    double2 *wa = W + blockIdx.y * p.w_map + (int64_t)ra * p.ldz;
    double2 *wb = W + blockIdx.y * p.w_map + (int64_t)(rb >= 0 ? rb : 0) * p.ldz;
    const double *ma = mask + (int64_t)ra * g.n2, *mb = mask + (int64_t)(rb >= 0 ? rb : 0) * g.n2;
    const int K = mp.kz_max;
    // element e of the packed line a + i b (Y left the planes kz = 0 and n / 2 real)
    auto ldf = [&](int e, int side) {
        const bool up = side ? side > 0 : 2 * e > n;
        const int kz = up ? n - e : e;
        double2 v = make_double2(0.0, 0.0);
        if (kz > K) return v;
        const double2 a = wa[kz];
        if (rb < 0) return make_double2(a.x, up ? -a.y : a.y);
        const double2 b = wb[kz];
        return up ? make_double2(a.x + b.y, b.x - a.y) : make_double2(a.x - b.y, a.y + b.x);
    };
    // F[e] of the forward transform: the rows hold F[kz] and i conj(F[n - kz])
    auto stf = [&](int e, double2 v, int side) {
        if (e <= p.kz_out) wa[e] = v;
        if (rb >= 0) {
            const int kz = side < 0 && e > 0 ? n : e == 0 ? 0 : n - e;  // (the lower half has only kz = 0)
            if (kz <= p.kz_out) wb[kz] = make_double2(v.y, v.x);
        }
    };
    auto ati = [&](int e) { return fft::row_at(ai, e); };
    auto atf = [&](int e) { return fft::row_at(af, e); };
    double2 *in = sm;
    if (ai.np >= 2) {
        if (on) fft::line_pass<double, 1, 0>(use_i, t, nt, twi, ldf, [&](int e, double2 v, int) { sm[ati(e)] = v; });
        __syncthreads();
    }
    if (ai.np == 3) {
        if (on)
            fft::line_pass<double, 1, 1>(use_i, t, nt, twi, [&](int e, int) { return sm[ati(e)]; },
                                         [&](int e, double2 v, int) { sm2[ati(e)] = v; });
        __syncthreads();
        in = sm2;
    }
    // last inverse pass, mask and first forward pass in registers: thread t holds z = t + r n / R
    const int q = ai.np - 1, nb = ai.nb[q];
    fft::with_last_radix(use_i, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        double2 v[R];
        const bool act = on && t < nb;
        if (act) {
            if (q == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = ldf(t + r * nb, 0);
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = in[ati(t + r * nb)];
                const double2 *w = twi + ai.tw[q] + t;
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = fft::mul_tw<1>(v[r], w[(r - 1) * nb]);
            }
            fft::Dft<R, 1, double, double2>::run(v);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                v[r].x *= ma[t + r * nb];
                if (rb >= 0) v[r].y *= mb[t + r * nb];
                else v[r] = make_double2(2.0 * v[r].x, 0.0);  // (the legs carry 1/2 for the unpacking of a pair)
            }
            fft::Dft<R, -1, double, double2>::run(v);
        }
        __syncthreads();  // the exchange buffer (and, for one pass, the rows in memory) have been read
        if (act) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (af.np == 1) stf(t + r, v[r], 0);
                else sm[atf(t * R + r)] = v[r];
            }
        }
    });
    if (af.np == 1) return;
    __syncthreads();
    if (af.np == 2) {
        if (on) fft::line_pass<double, -1, 1>(use_f, t, nt, twf, [&](int e, int) { return sm[atf(e)]; }, stf);
        return;
    }
    if (on)
        fft::line_pass<double, -1, 1>(use_f, t, nt, twf, [&](int e, int) { return sm[atf(e)]; },
                                      [&](int e, double2 v, int) { sm2[atf(e)] = v; });
    __syncthreads();
    if (on) fft::line_pass<double, -1, 2>(use_f, t, nt, twf, [&](int e, int) { return sm2[atf(e)]; }, stf);
}

// ---- products: forward transform along z of X_i Y_j - Z_i Z_j, two rows per complex line ----------
// block (threads per line, L pairs of rows); grid (products, row pairs / L): the products of a few rows follow each
// other, so the maps' rows come from L2 after the first.  The row blocks lie in y and z: those of 512 x 512 x 500 and of
// 640^3 are more than y takes (in x with the products, taken apart by a division, 5 products of 150 x 135 x 144 took 104
// against 101 us)
struct MrPairs {
    int16_t i[MR_MAX_MAPS], j[MR_MAX_MAPS];
};
template <int N>
__global__ void __launch_bounds__(MR_THREADS, 2) mr_product_kernel(const __grid_constant__ MrParams p,
                                                                  const __grid_constant__ MrPairs pr,
                                                                  const double2 *table, const double *X, const double *Y,
                                                                  const double *Z, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const fft::AxisUse<N, true> use(p.azf);
    const Axis &ax = use.v;
    const int L = blockDim.y, n = ax.n, ld = fft::row_len(ax);
    double2 *tw = mr_smem, *sm = tw + ax.tw_len + threadIdx.y * ld, *sm2 = sm + L * ld;
    load_table(tw, table + p.tw_zf, ax.tw_len);
    const int half = (g.n1 + 1) / 2, q = (blockIdx.z * gridDim.y + blockIdx.y) * L + threadIdx.y;
    const bool on = q < g.n0 * half;
    const int x = on ? q / half : 0, y = on ? 2 * (q - x * half) : 0;
    const bool two = y + 1 < g.n1;
    const double h = two ? 0.5 : 1.0;
    const int64_t ra = (int64_t)x * g.n1 + y, oi = pr.i[blockIdx.x] * g.nreal, oj = pr.j[blockIdx.x] * g.nreal;
    const double *xi = X + oi + ra * n, *xj = Y + oj + ra * n;
    const double *zi = Z ? Z + oi + ra * n : nullptr, *zj = Z ? Z + oj + ra * n : nullptr;
    double2 *wa = W + blockIdx.x * p.w_map + ra * p.ldz, *wb = wa + p.ldz;
    fft::line_fft<double, -1>(
        use, threadIdx.x, N ? ax.nb[0] : (int)blockDim.x, on, sm, sm2, tw, [&](int e) { return fft::row_at(ax, e); },
        [&](int e, int) {
            double2 v = make_double2(xi[e] * xj[e], 0.0);
            if (Z) v.x -= zi[e] * zj[e];
            if (two) {
                v.y = xi[e + n] * xj[e + n];
                if (Z) v.y -= zi[e + n] * zj[e + n];
            }
            v.x *= h;
            v.y *= h;
            return v;
        },
        [&](int e, double2 v, int side) {
            if (e <= p.kz_out) wa[e] = v;
            const int kz = side < 0 && e > 0 ? n : e == 0 ? 0 : n - e;
            if (two && kz <= p.kz_out) wb[kz] = make_double2(v.y, v.x);
        });
}

// ---- X': forward transform along x ---------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_out_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                              const int32_t *x_on, const double2 *W, double2 *out) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const fft::AxisUse<N, true> use(p.ax);
    const Axis &ax = use.v;
    const int L = N ? line_count(ax) : blockDim.x, NT = N ? line_threads(ax) : blockDim.y, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, g.n1);
    if (abs(ky) > ky_radius(g, p.out2, kz0)) return;
    double2 *tw = mr_smem, *sm = tw + ax.tw_len, *sm2 = sm + ax.n * L;
    load_table(tw, table + p.tw_x, ax.tw_len);
    const int line = threadIdx.x, kz = kz0 + line;
    const bool on = kz <= p.kz_out;
    const double2 *w = W + blockIdx.y * p.w_map + (int64_t)iy * p.ldz + kz;
    const int wx = g.n1 * p.ldz * (int)sizeof(double2), ox = g.n1 * g.nh2 * (int)sizeof(double2);
    double2 *o = out + blockIdx.y * g.nhalf + (int64_t)iy * g.nh2 + kz;
    const int rx = index_radius(p.out2, (ky * g.kf1) * (ky * g.kf1) + (kz * g.kf2) * (kz * g.kf2), g.kf0);
    fft::line_fft<double, -1>(
        use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int x, int) { return !x_on || x_on[x] ? elem(w, x, wx) : make_double2(0.0, 0.0); },
        [&](int e, double2 v, int side) {
            if (fft::abs_label(e, ax.n, side) <= rx) elem(o, e, ox) = v;
        });
}

// ---- launches ---------------------------------------------------------------------------------
struct MrShapes {
    int Lx, Tx, Ly, Ty, Lz, Tz;   // lines per block and threads per line of each axis
    size_t sx, sy, sz;
};
struct MrArgs {
    const double2 *src, *table;
    const double *mask, *X, *Y, *Z;
    const int32_t *pairs, *xs, *x_on;
    const uint8_t *pair_on;
    double2 *W, *out;
    int maps;
    MrPairs products;
};
enum MrStage { MR_X, MR_Y, MR_Z, MR_PRODUCT, MR_Y_BACK, MR_X_BACK };

// blocks of a stage for nm maps
struct MrGrid {
    int64_t x, y, z;
};
static inline MrGrid mr_grid(MrStage stage, const MrParams &p, const MrShapes &sh, int nm) {
    switch (stage) {
        case MR_X:
        case MR_X_BACK: return {(int64_t)p.g.n1 * (p.kz_out / sh.Lx + 1), nm, 1};
        case MR_Y:
        case MR_Y_BACK: return {(int64_t)p.n_x * (p.kz_out / sh.Ly + 1), nm, 1};
        case MR_Z: return {((int64_t)p.n_pairs + sh.Lz - 1) / sh.Lz, nm, 1};
        default: {
            const int64_t rows = ((int64_t)p.g.n0 * ((p.g.n1 + 1) / 2) + sh.Lz - 1) / sh.Lz, z = (rows + 65534) / 65535;
            return {nm, (rows + z - 1) / z, z};
        }
    }
}

template <typename K> static cudaError_t mr_allow(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// one stage of the nm maps in W with the kernels of length N (0: the run-time plan)
template <int N>
cudaError_t mr_launch(MrStage stage, const MrParams &p, const MrShapes &sh, const MrArgs &a, cudaStream_t s) {
    const MrGrid n = mr_grid(stage, p, sh, a.maps);
    const dim3 grid((unsigned)n.x, (unsigned)n.y, (unsigned)n.z);
    cudaError_t e = cudaSuccess;
    switch (stage) {
        case MR_X:
            if ((e = mr_allow(mr_x_kernel<N>, sh.sx)) != cudaSuccess) return e;
            mr_x_kernel<N><<<grid, dim3(sh.Lx, sh.Tx), sh.sx, s>>>(p, a.src, a.table, a.W);
            break;
        case MR_Y:
            if ((e = mr_allow(mr_y_kernel<1, N>, sh.sy)) != cudaSuccess) return e;
            mr_y_kernel<1, N><<<grid, dim3(sh.Ly, sh.Ty), sh.sy, s>>>(p, a.table, a.xs, a.pair_on, a.W);
            break;
        case MR_Z:
            if ((e = mr_allow(mr_z_kernel<N>, sh.sz)) != cudaSuccess) return e;
            mr_z_kernel<N><<<grid, dim3(sh.Tz, sh.Lz), sh.sz, s>>>(p, a.table, a.pairs, a.mask, a.W);
            break;
        case MR_PRODUCT:
            if ((e = mr_allow(mr_product_kernel<N>, sh.sz)) != cudaSuccess) return e;
            mr_product_kernel<N><<<grid, dim3(sh.Tz, sh.Lz), sh.sz, s>>>(p, a.products, a.table, a.X, a.Y, a.Z, a.W);
            break;
        case MR_Y_BACK:
            if ((e = mr_allow(mr_y_kernel<-1, N>, sh.sy)) != cudaSuccess) return e;
            mr_y_kernel<-1, N><<<grid, dim3(sh.Ly, sh.Ty), sh.sy, s>>>(p, a.table, a.xs, a.pair_on, a.W);
            break;
        case MR_X_BACK:
            if ((e = mr_allow(mr_out_kernel<N>, sh.sx)) != cudaSuccess) return e;
            mr_out_kernel<N><<<grid, dim3(sh.Lx, sh.Tx), sh.sx, s>>>(p, a.table, a.x_on, a.W, a.out);
            break;
    }
    return cudaGetLastError();
}

// Lengths with kernels of their own (radices, strides and counts known to the compiler): twenty even lengths from 48 to
// 256 with factors 2, 3 and 5, not all of them (each costs three families of kernels seconds of compilation).  Every
// other length, 50, 54, 162, 250 and the odd ones among them, runs the run-time plan.
// 60 rows of 128^3 on a ball mask: 1.23 ms against 1.59 ms with the run-time plan, 78 products 1.06
// against 1.72 ms.  The groups only spread the compilation over files.
#define MR_GROUP_0(X) X(48) X(60) X(64) X(72) X(80)
#define MR_GROUP_1(X) X(90) X(96) X(100) X(108) X(120)
#define MR_GROUP_2(X) X(128) X(144) X(150) X(160) X(180)
#define MR_GROUP_3(X) X(192) X(200) X(216) X(240) X(256)
#define MR_CASE(N) \
    case N: *e = mr_launch<N>(stage, p, sh, a, s); return true;
// true when the group holds length n (and launched the stage)
#define MR_DEFINE_GROUP(K)                                                                                   \
    bool mr_group_##K(int n, MrStage stage, const MrParams &p, const MrShapes &sh, const MrArgs &a,          \
                      cudaStream_t s, cudaError_t *e) {                                                      \
        switch (n) { MR_GROUP_##K(MR_CASE) }                                                                 \
        return false;                                                                                        \
    }
#define MR_DECLARE_GROUP(K)                                                                                  \
    bool mr_group_##K(int n, MrStage stage, const MrParams &p, const MrShapes &sh, const MrArgs &a,          \
                      cudaStream_t s, cudaError_t *e);
MR_DECLARE_GROUP(0)
MR_DECLARE_GROUP(1)
MR_DECLARE_GROUP(2)
MR_DECLARE_GROUP(3)

}  // namespace pb
