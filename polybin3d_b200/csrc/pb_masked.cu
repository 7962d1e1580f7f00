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
// W holds kz <= k_out / kF only.  Bound by FP64 and integer issue (16 warps per SM at 128 registers)
// rather than by memory: chunks of 5 maps whose W stays in L2 took longer (1.48 ms) than chunks of
// 32 (more blocks per launch, fewer tails).
// Measured on a B200, 60 rows of 128^3 (bins to 0.93 of the Nyquist frequency), against 2.95 ms for
// filter, cuFFT and mask: 0.97 ms on a sector mask (17 % of the rows), 1.89 ms on a ball (71 %).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>
#include "pb_fft.cuh"

namespace pb {
namespace fft {

static int balanced_radix(int n) {
    // n = R0 R1 with both radices at most 16 and R0 <= R1 as large as possible; 0 when impossible
    for (int r = 16; r >= 2; --r)
        if (n % r == 0 && n / r <= MAX_RADIX && n / r >= r) return r;
    return 0;
}

bool plan_axis(int n, bool reversed, Axis *ax) {
    memset(ax, 0, sizeof(*ax));
    if (n < 2 || n > 1024) return false;
    ax->n = n;
    int r[3] = {n, 0, 0};
    if (n <= MAX_RADIX) {
        ax->np = 1;
    } else if (int a = balanced_radix(n)) {
        ax->np = 2;
        r[0] = a;
        r[1] = n / a;
    } else {
        // three passes: the largest last radix whose cofactor splits in two
        ax->np = 0;
        for (int c = MAX_RADIX; c >= 2 && !ax->np; --c) {
            if (n % c) continue;
            const int b = balanced_radix(n / c);
            if (b && n / c / b <= c) {
                ax->np = 3;
                r[0] = b;
                r[1] = n / c / b;
                r[2] = c;
            }
        }
        if (!ax->np) return false;
    }
    if (reversed) std::reverse(r, r + ax->np);
    int ns = 1;
    for (int q = 0; q < ax->np; ++q) {
        ax->R[q] = r[q];
        ax->nb[q] = n / r[q];
        ax->ns[q] = ns;
        ax->tw[q] = ax->tw_len;
        if (q > 0) ax->tw_len += (r[q] - 1) * ns;
        ns *= r[q];
    }
    ax->div_ns1 = ((1u << 20) + (uint32_t)r[0] - 1) / (uint32_t)r[0];
    ax->pad = (r[0] % 2 == 0) ? 1 : 0;
    return true;
}

void fill_twiddles(const Axis &ax, double *out) {
    for (int q = 1; q < ax.np; ++q) {
        const int ns = ax.ns[q], len = ns * ax.R[q];
        for (int r = 1; r < ax.R[q]; ++r)
            for (int jm = 0; jm < ns; ++jm) {
                const long double a = 2.0L * 3.14159265358979323846264338327950288L * (r * jm) / len;
                double *o = out + 2 * (ax.tw[q] + (r - 1) * ns + jm);
                o[0] = (double)cosl(a);
                o[1] = (double)sinl(a);
            }
    }
}

}  // namespace fft

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
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_x_kernel(const __grid_constant__ MrParams p, const double2 *src,
                                                            const double2 *table, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const int L = blockDim.x, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, g.n1);
    if (kz0 > mp.kz_max || abs(ky) > ky_radius(g, mp.hi2, kz0)) return;
    double2 *tw = mr_smem, *sm = tw + p.ax.tw_len, *sm2 = sm + p.ax.n * L;
    load_table(tw, table + p.tw_x, p.ax.tw_len);
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
        p.ax, threadIdx.y, blockDim.y, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int e) {
            double2 v = make_double2(0.0, 0.0);
            const int kx = freq_index(e, g.n0), ax = abs(kx);
            if (ax > r_out || ax < r_in) return v;
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
        [&](int x, double2 v) { elem(w, x, wx) = v; });
}

// ---- Y: inverse (SIGN 1) and forward (SIGN -1) transforms along y, in place ---------------
// Rows go in pairs (y even, y + 1), the last one alone when n1 is odd; pair_on[x ceil(n1 / 2) + y / 2]:
// the mask is not zero on both (NULL: every pair).  xs: the planes x to do (NULL: all).
template <int SIGN>
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_y_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                            const int32_t *xs, const uint8_t *pair_on, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const int L = blockDim.x, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, xi = blockIdx.x / runs, x = xs ? xs[xi] : xi,
              kz0 = run * L;
    const int kz_max = SIGN > 0 ? mp.kz_max : p.kz_out;
    if (kz0 > kz_max) return;
    double2 *tw = mr_smem, *sm = tw + p.ay.tw_len, *sm2 = sm + p.ay.n * L;
    load_table(tw, table + p.tw_y, p.ay.tw_len);
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
    if (SIGN > 0) {
        fft::line_fft<double, 1>(
            p.ay, threadIdx.y, blockDim.y, on, sm, sm2, tw, at,
            [&](int e) { return abs(freq_index(e, g.n1)) <= ry ? elem(w, e, row) : zero; },
            [&](int y, double2 v) {
                if (act[y >> 1]) elem(w, y, row) = v;
            });
    } else {
        // With F the packed transform of a pair (halved on its way in), row y even holds F[kz] and row
        // y + 1 holds i conj(F[-kz]): the transform of either row is then own - i other.  The other
        // comes from the lane 16 further where that lane reads row y ^ 1 in the same round
        const bool shuffle = L == 16 && (p.ay.nb[0] & 1) == 0 && (g.n1 & 1) == 0;
        const unsigned lanes = __ballot_sync(0xffffffffu, on);
        fft::line_fft<double, -1>(
            p.ay, threadIdx.y, blockDim.y, on, sm, sm2, tw, at,
            [&](int y) { return act[y >> 1] ? elem(w, y, row) : zero; },
            [&](int e, double2 v) {
                if (abs(freq_index(e, g.n1)) <= ry) elem(w, e, row) = v;
            },
            [&](int y, double2 v) {
                double2 o;
                if (shuffle) {
                    o.x = __shfl_xor_sync(lanes, v.x, 16);
                    o.y = __shfl_xor_sync(lanes, v.y, 16);
                } else {
                    if ((y ^ 1) >= g.n1) return v;
                    o = act[y >> 1] ? elem(w, y ^ 1, row) : zero;
                }
                return make_double2(v.x + o.y, v.y - o.x);
            });
    }
}

// ---- Z: inverse transform along z, mask, forward transform -------------------------------
// block (threads per line = butterflies of the last inverse pass, L pairs of rows); grid (pairs / L, maps)
__global__ void __launch_bounds__(MR_THREADS, 2) mr_z_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                            const int32_t *pairs, const double *mask, double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const MrMap &mp = p.maps[blockIdx.y];
    const Axis &ai = p.azi, &af = p.azf;
    const int L = blockDim.y, t = threadIdx.x, nt = blockDim.x, n = ai.n;
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
    // element e of the packed line a + i b; the planes kz = 0 and n / 2 are real
    auto ldf = [&](int e) {
        const bool up = 2 * e > n;
        const int kz = up ? n - e : e;
        double2 v = make_double2(0.0, 0.0);
        if (kz > K) return v;
        const double2 a = wa[kz];
        const double2 b = rb >= 0 ? wb[kz] : v;
        if (kz == 0 || 2 * kz == n) return make_double2(a.x, b.x);
        return up ? make_double2(a.x + b.y, b.x - a.y) : make_double2(a.x - b.y, a.y + b.x);
    };
    // F[e] of the forward transform: the rows hold F[kz] and i conj(F[n - kz])
    auto stf = [&](int e, double2 v) {
        if (e <= p.kz_out) wa[e] = v;
        if (rb >= 0) {
            const int kz = e == 0 ? 0 : n - e;
            if (kz <= p.kz_out) wb[kz] = make_double2(v.y, v.x);
        }
    };
    auto ati = [&](int e) { return fft::row_at(ai, e); };
    auto atf = [&](int e) { return fft::row_at(af, e); };
    double2 *in = sm;
    if (ai.np >= 2) {
        if (on) fft::line_pass<double, 1, 0>(ai, t, nt, twi, ldf, [&](int e, double2 v) { sm[ati(e)] = v; });
        __syncthreads();
    }
    if (ai.np == 3) {
        if (on)
            fft::line_pass<double, 1, 1>(ai, t, nt, twi, [&](int e) { return sm[ati(e)]; },
                                         [&](int e, double2 v) { sm2[ati(e)] = v; });
        __syncthreads();
        in = sm2;
    }
    // last inverse pass, mask and first forward pass in registers: thread t holds z = t + r n / R
    const int q = ai.np - 1, nb = ai.nb[q];
    fft::with_radix(ai.R[q], [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        double2 v[R];
        const bool act = on && t < nb;
        if (act) {
            if (q == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = ldf(t + r * nb);
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
                if (af.np == 1) stf(t + r, v[r]);
                else sm[atf(t * R + r)] = v[r];
            }
        }
    });
    if (af.np == 1) return;
    __syncthreads();
    if (af.np == 2) {
        if (on) fft::line_pass<double, -1, 1>(af, t, nt, twf, [&](int e) { return sm[atf(e)]; }, stf);
        return;
    }
    if (on)
        fft::line_pass<double, -1, 1>(af, t, nt, twf, [&](int e) { return sm[atf(e)]; },
                                      [&](int e, double2 v) { sm2[atf(e)] = v; });
    __syncthreads();
    if (on) fft::line_pass<double, -1, 2>(af, t, nt, twf, [&](int e) { return sm2[atf(e)]; }, stf);
}

// ---- products: forward transform along z of X_i X_j - Z_i Z_j, two rows per complex line ----------
// block (threads per line, L pairs of rows); grid (products, row pairs / L): the products of a few
// rows follow each other, so the maps' rows come from L2 after the first
struct MrPairs {
    int16_t i[MR_MAX_MAPS], j[MR_MAX_MAPS];
};
__global__ void __launch_bounds__(MR_THREADS, 2) mr_product_kernel(const __grid_constant__ MrParams p,
                                                                  const __grid_constant__ MrPairs pr,
                                                                  const double2 *table, const double *X, const double *Z,
                                                                  double2 *W) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const Axis &ax = p.azf;
    const int L = blockDim.y, n = ax.n, ld = fft::row_len(ax);
    double2 *tw = mr_smem, *sm = tw + ax.tw_len + threadIdx.y * ld, *sm2 = sm + L * ld;
    load_table(tw, table + p.tw_zf, ax.tw_len);
    const int half = (g.n1 + 1) / 2, q = blockIdx.y * L + threadIdx.y;
    const bool on = q < g.n0 * half;
    const int x = on ? q / half : 0, y = on ? 2 * (q - x * half) : 0;
    const bool two = y + 1 < g.n1;
    const double h = two ? 0.5 : 1.0;
    const int64_t ra = (int64_t)x * g.n1 + y, oi = pr.i[blockIdx.x] * g.nreal, oj = pr.j[blockIdx.x] * g.nreal;
    const double *xi = X + oi + ra * n, *xj = X + oj + ra * n;
    const double *zi = Z ? Z + oi + ra * n : nullptr, *zj = Z ? Z + oj + ra * n : nullptr;
    double2 *wa = W + blockIdx.x * p.w_map + ra * p.ldz, *wb = wa + p.ldz;
    fft::line_fft<double, -1>(
        ax, threadIdx.x, blockDim.x, on, sm, sm2, tw, [&](int e) { return fft::row_at(ax, e); },
        [&](int e) {
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
        [&](int e, double2 v) {
            if (e <= p.kz_out) wa[e] = v;
            const int kz = e == 0 ? 0 : n - e;
            if (two && kz <= p.kz_out) wb[kz] = make_double2(v.y, v.x);
        });
}

// ---- X': forward transform along x ---------------------------------------------------------
__global__ void __launch_bounds__(MR_LINE_THREADS, 5) mr_out_kernel(const __grid_constant__ MrParams p, const double2 *table,
                                                              const int32_t *x_on, const double2 *W, double2 *out) {
    extern __shared__ __align__(16) double2 mr_smem[];
    const Grid &g = p.g;
    const int L = blockDim.x, runs = p.kz_out / L + 1;
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, g.n1);
    if (abs(ky) > ky_radius(g, p.out2, kz0)) return;
    double2 *tw = mr_smem, *sm = tw + p.ax.tw_len, *sm2 = sm + p.ax.n * L;
    load_table(tw, table + p.tw_x, p.ax.tw_len);
    const int line = threadIdx.x, kz = kz0 + line;
    const bool on = kz <= p.kz_out;
    const double2 *w = W + blockIdx.y * p.w_map + (int64_t)iy * p.ldz + kz;
    const int wx = g.n1 * p.ldz * (int)sizeof(double2), ox = g.n1 * g.nh2 * (int)sizeof(double2);
    double2 *o = out + blockIdx.y * g.nhalf + (int64_t)iy * g.nh2 + kz;
    const int rx = index_radius(p.out2, (ky * g.kf1) * (ky * g.kf1) + (kz * g.kf2) * (kz * g.kf2), g.kf0);
    fft::line_fft<double, -1>(
        p.ax, threadIdx.y, blockDim.y, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int x) { return !x_on || x_on[x] ? elem(w, x, wx) : make_double2(0.0, 0.0); },
        [&](int e, double2 v) {
            if (abs(freq_index(e, g.n0)) <= rx) elem(o, e, ox) = v;
        });
}

// ---- host side ------------------------------------------------------------------------------
struct MrLayout {
    Axis ax, ay, azi, azf;
    int tw_x, tw_y, tw_zi, tw_zf, tw_len;
};

static int mr_layout(const Grid &G, MrLayout *L) {
    // the larger radix where the operands come from memory: all of a thread's loads in one round
    if (!fft::plan_axis(G.n0, true, &L->ax) || !fft::plan_axis(G.n1, true, &L->ay) ||
        !fft::plan_axis(G.n2, false, &L->azi) || !fft::plan_axis(G.n2, true, &L->azf))
        return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: grid dimensions must be products of 2, 3, 5, 7, 11 and 13 "
                                        "of at most three factors up to 16");
    L->tw_x = 0;
    L->tw_y = L->tw_x + L->ax.tw_len;
    L->tw_zi = L->tw_y + L->ay.tw_len;
    L->tw_zf = L->tw_zi + L->azi.tw_len;
    L->tw_len = L->tw_zf + L->azf.tw_len;
    return PB_OK;
}

static int mr_row_stride(const Grid &G, double k_out) {
    const int kz = std::min(G.nh2 - 1, (int)std::floor(k_out / G.kf2));
    return (kz + 8) & ~7;  // rows of whole 128-byte lines
}

// lines per block and threads per line of an x / y transform, and its shared memory
static void line_shape(const Axis &ax, int *L, int *nt, size_t *smem) {
    const int bufs = ax.np - 1;
    *L = ax.np == 1 ? 32 : 16;
    auto bytes = [&](int l) { return ((size_t)ax.tw_len + (size_t)bufs * l * ax.n) * sizeof(double2); };
    while (*L > 2 && bytes(*L) > (size_t)MR_SMEM) *L /= 2;
    *nt = std::max(1, std::min(ax.nb[0], MR_LINE_THREADS / *L));
    *smem = bytes(*L);
}

struct MrShapes {
    int Lx, Tx, Ly, Ty, Lz, Tz;   // lines per block and threads per line of each axis
    size_t sx, sy, sz;
};

// everything of MrParams that the grid and k_out fix, and the launch shapes
static int mr_setup(const Grid &G, double k_out, MrParams *pp, MrShapes *sh) {
    MrLayout lay;
    const int st = mr_layout(G, &lay);
    if (st) return st;
    MrParams &p = *pp;
    memset(&p, 0, sizeof(p));
    p.g = G;
    p.ldz = mr_row_stride(G, k_out);
    p.kz_out = std::min(G.nh2 - 1, (int)std::floor(k_out / G.kf2));
    p.out2 = k_out * k_out * (1.0 + 1e-12);
    p.w_map = (int64_t)G.n0 * G.n1 * p.ldz;
    p.ax = lay.ax;
    p.ay = lay.ay;
    p.azi = lay.azi;
    p.azf = lay.azf;
    p.tw_x = lay.tw_x;
    p.tw_y = lay.tw_y;
    p.tw_zi = lay.tw_zi;
    p.tw_zf = lay.tw_zf;
    line_shape(p.ax, &sh->Lx, &sh->Tx, &sh->sx);
    line_shape(p.ay, &sh->Ly, &sh->Ty, &sh->sy);
    // z: one butterfly of the last inverse pass per thread, pairs of rows up to 128 threads
    const int Tz = p.azi.nb[p.azi.np - 1];
    const int ldr = std::max(fft::row_len(p.azi), fft::row_len(p.azf));
    auto zbytes = [&](int l) {
        return ((size_t)p.azi.tw_len + p.azf.tw_len + (size_t)(p.azi.np == 3 ? 2 : 1) * l * ldr) * sizeof(double2);
    };
    int Lz = std::max(1, 128 / Tz);
    while (Lz > 1 && zbytes(Lz) > (size_t)MR_SMEM) Lz /= 2;
    sh->Lz = Lz;
    sh->Tz = Tz;
    sh->sz = zbytes(Lz);
    if (Tz * Lz > MR_THREADS || std::max(sh->sz, std::max(sh->sx, sh->sy)) > (size_t)MR_SMEM)
        return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: lines too long");
    return PB_OK;
}

static double threshold_sq(double e) {  // smallest t with sqrt(t) >= e
    if (!(e > 0.0)) return 0.0;
    double t = e * e;
    while (t > 0.0 && std::sqrt(t) >= e) t = std::nextafter(t, 0.0);
    while (std::sqrt(t) < e) t = std::nextafter(t, HUGE_VAL);
    return t;
}

}  // namespace pb

using namespace pb;

extern "C" int pb_masked_rows_table(const pb_grid_t *g, double *table, size_t *bytes) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!bytes) return fail(PB_ERR_INVALID, "pb_masked_rows_table: bytes is NULL");
    MrLayout L;
    st = mr_layout(G, &L);
    if (st) return st;
    const size_t need = std::max<size_t>(16, (size_t)L.tw_len * 16);
    if (table) {
        if (*bytes < need) return fail(PB_ERR_INVALID, "pb_masked_rows_table: buffer too small");
        fft::fill_twiddles(L.ax, table + 2 * L.tw_x);
        fft::fill_twiddles(L.ay, table + 2 * L.tw_y);
        fft::fill_twiddles(L.azi, table + 2 * L.tw_zi);
        fft::fill_twiddles(L.azf, table + 2 * L.tw_zf);
    }
    *bytes = need;
    return PB_OK;
}

extern "C" int pb_masked_rows_workspace_size(const pb_grid_t *g, double k_out, int n_maps, size_t *bytes) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!bytes || n_maps < 1 || !(k_out > 0.0)) return fail(PB_ERR_INVALID, "pb_masked_rows_workspace_size: bad argument");
    MrLayout L;
    st = mr_layout(G, &L);
    if (st) return st;
    *bytes = (size_t)std::min(n_maps, MR_MAX_MAPS) * G.n0 * G.n1 * mr_row_stride(G, k_out) * sizeof(double2);
    return PB_OK;
}

extern "C" int pb_masked_rows(const pb_grid_t *g, const void *src, int64_t src_stride, int n_maps, int n_legs,
                              const int32_t *src_idx, const double *lo, const double *hi, const int32_t *ell,
                              const double *scale, double k_out, const double *mask, const int32_t *pairs, int n_pairs,
                              const uint8_t *pair_on, const int32_t *xs, int n_x, const int32_t *x_on,
                              const void *table, void *out, void *workspace, size_t workspace_bytes, void *stream) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!src || !src_idx || !lo || !hi || !ell || !scale || !mask || !pairs || !pair_on || !xs || !x_on || !table || !out)
        return fail(PB_ERR_INVALID, "pb_masked_rows: NULL argument");
    if (n_maps < 1 || n_legs < 1 || n_legs > MR_MAX_LEGS || n_pairs < 1 || n_x < 1 || n_x > G.n0 || !(k_out > 0.0))
        return fail(PB_ERR_INVALID, "pb_masked_rows: bad sizes");
    MrParams p;
    MrShapes sh;
    st = mr_setup(G, k_out, &p, &sh);
    if (st) return st;
    p.n_legs = n_legs;
    p.src_stride = src_stride;
    p.n_x = n_x;
    p.n_pairs = n_pairs;
    for (int i = 0; i < n_maps * n_legs; ++i) {
        if (ell[i] != 0 && ell[i] != 2 && ell[i] != 4) return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: even Legendre orders up to 4");
        if (ell[i] != 0 && G.los) return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: Legendre weights need the global line of sight");
        if (src_idx[i] < 0) return fail(PB_ERR_INVALID, "pb_masked_rows: negative source index");
        if (!(hi[i] > 0.0) || hi[i] > k_out) return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: upper edges must lie in (0, k_out]");
    }
    const size_t per = (size_t)p.w_map * sizeof(double2);
    const int chunk = (int)std::min<size_t>(MR_MAX_MAPS, workspace_bytes / per);
    if (!workspace || chunk < 1) return fail(PB_ERR_WORKSPACE, "pb_masked_rows: workspace too small");
    PB_CUDA(cudaFuncSetAttribute(mr_x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sx));
    PB_CUDA(cudaFuncSetAttribute(mr_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sx));
    PB_CUDA(cudaFuncSetAttribute(mr_y_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sy));
    PB_CUDA(cudaFuncSetAttribute(mr_y_kernel<-1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sy));
    PB_CUDA(cudaFuncSetAttribute(mr_z_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sz));
    cudaStream_t s = as_stream(stream);
    double2 *W = (double2 *)workspace;
    const double2 *tab = (const double2 *)table;
    for (int m0 = 0; m0 < n_maps; m0 += chunk) {
        const int nm = std::min(chunk, n_maps - m0);
        for (int m = 0; m < nm; ++m) {
            MrMap &mp = p.maps[m];
            double top = 0.0, low = HUGE_VAL;
            for (int q = 0; q < n_legs; ++q) {
                const int i = (m0 + m) * n_legs + q;
                mp.leg[q] = MrLeg{threshold_sq(lo[i]), threshold_sq(hi[i]), 0.5 * scale[i], src_idx[i], ell[i]};
                top = std::max(top, hi[i]);
                low = std::min(low, std::max(lo[i], 0.0));
            }
            mp.hi2 = top * top * (1.0 + 1e-12);
            mp.lo2 = low * low;
            mp.kz_max = std::min(p.kz_out, (int)std::floor(top / G.kf2));
        }
        const int runs_x = p.kz_out / sh.Lx + 1, runs_y = p.kz_out / sh.Ly + 1;
        mr_x_kernel<<<dim3(G.n1 * runs_x, nm), dim3(sh.Lx, sh.Tx), sh.sx, s>>>(p, (const double2 *)src, tab, W);
        PB_LAUNCH_CHECK("pb_masked_rows(x)");
        mr_y_kernel<1><<<dim3(n_x * runs_y, nm), dim3(sh.Ly, sh.Ty), sh.sy, s>>>(p, tab, xs, pair_on, W);
        PB_LAUNCH_CHECK("pb_masked_rows(y)");
        mr_z_kernel<<<dim3((n_pairs + sh.Lz - 1) / sh.Lz, nm), dim3(sh.Tz, sh.Lz), sh.sz, s>>>(p, tab, pairs, mask, W);
        PB_LAUNCH_CHECK("pb_masked_rows(z)");
        mr_y_kernel<-1><<<dim3(n_x * runs_y, nm), dim3(sh.Ly, sh.Ty), sh.sy, s>>>(p, tab, xs, pair_on, W);
        PB_LAUNCH_CHECK("pb_masked_rows(y')");
        mr_out_kernel<<<dim3(G.n1 * runs_x, nm), dim3(sh.Lx, sh.Tx), sh.sx, s>>>(p, tab, x_on, W,
                                                                                 (double2 *)out + (int64_t)m0 * G.nhalf);
        PB_LAUNCH_CHECK("pb_masked_rows(x')");
    }
    return PB_OK;
}

extern "C" int pb_product_rows(const pb_grid_t *g, const double *X, const double *Z, const int32_t *pairs, int n_pairs,
                               double k_out, const void *table, void *out, void *workspace, size_t workspace_bytes,
                               void *stream) {
    Grid G;
    int st = make_grid(g, &G);
    if (st) return st;
    if (!X || !pairs || !table || !out) return fail(PB_ERR_INVALID, "pb_product_rows: NULL argument");
    if (n_pairs < 1 || !(k_out > 0.0)) return fail(PB_ERR_INVALID, "pb_product_rows: bad sizes");
    for (int k = 0; k < 2 * n_pairs; ++k)
        if (pairs[k] < 0 || pairs[k] > 32767) return fail(PB_ERR_INVALID, "pb_product_rows: map index out of range");
    MrParams p;
    MrShapes sh;
    st = mr_setup(G, k_out, &p, &sh);
    if (st) return st;
    const size_t per = (size_t)p.w_map * sizeof(double2);
    const int chunk = (int)std::min<size_t>(MR_MAX_MAPS, workspace_bytes / per);
    if (!workspace || chunk < 1) return fail(PB_ERR_WORKSPACE, "pb_product_rows: workspace too small");
    PB_CUDA(cudaFuncSetAttribute(mr_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sz));
    PB_CUDA(cudaFuncSetAttribute(mr_y_kernel<-1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sy));
    PB_CUDA(cudaFuncSetAttribute(mr_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.sx));
    cudaStream_t s = as_stream(stream);
    double2 *W = (double2 *)workspace;
    const double2 *tab = (const double2 *)table;
    const int rows = G.n0 * ((G.n1 + 1) / 2);
    for (int m0 = 0; m0 < n_pairs; m0 += chunk) {
        const int nm = std::min(chunk, n_pairs - m0);
        MrPairs pr;
        for (int m = 0; m < nm; ++m) {
            pr.i[m] = (int16_t)pairs[2 * (m0 + m)];
            pr.j[m] = (int16_t)pairs[2 * (m0 + m) + 1];
        }
        mr_product_kernel<<<dim3(nm, (rows + sh.Lz - 1) / sh.Lz), dim3(sh.Tz, sh.Lz), sh.sz, s>>>(p, pr, tab, X, Z, W);
        PB_LAUNCH_CHECK("pb_product_rows(z)");
        mr_y_kernel<-1><<<dim3(G.n0 * (p.kz_out / sh.Ly + 1), nm), dim3(sh.Ly, sh.Ty), sh.sy, s>>>(p, tab, nullptr,
                                                                                                  nullptr, W);
        PB_LAUNCH_CHECK("pb_product_rows(y)");
        mr_out_kernel<<<dim3(G.n1 * (p.kz_out / sh.Lx + 1), nm), dim3(sh.Lx, sh.Tx), sh.sx, s>>>(
            p, tab, nullptr, W, (double2 *)out + (int64_t)m0 * G.nhalf);
        PB_LAUNCH_CHECK("pb_product_rows(x)");
    }
    return PB_OK;
}
