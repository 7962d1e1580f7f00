// Legs of a gradient (pb_leg_gather): the adjoint of the map synthesis,
//   grad[dst_m](k) += scale_m Theta(lo_m <= |k| < hi_m) L_lm(mu) sum_x R[m](x) e^{-2 pi i k.x / M},
// in three passes over W[map][x][y][kz] (layout, lengths and bands of pb_synth_lines.cuh):
//   Z  per (map, pairs of rows): two real rows as one complex line, forward transform along z, the two
//      half spectra taken apart through shared memory, kz <= the map's band
//   Y  per (map, x, run of kz): forward transform along y in place, rows ky inside the band
//   X  per (ky in the band, run of kz, shell): forward transform along x of the maps of the shell in turn, each
//      filtered and added to the gradient (the shells are disjoint, so that no two blocks meet in a mode and
//      the order is fixed; 2 of 127 modes of a column lie in one shell, so the additions are few)
// cuFFT transformed every line of every map and wrote whole half spectra that the filter read back.
// Measured on a B200, the 32 legs of a 256^3 gradient (16 bins, l = 0, 2) on 192^3, FP32: 725 us against 1565 us for
// cuFFT and the filter.
#pragma once
#include "pb_synth_lines.cuh"

namespace pb {

// maps of shell q: order[first[q]] .. order[first[q + 1] - 1]
struct FlShells {
    int32_t n, first[SL_MAX_MAPS + 1];
    int8_t order[SL_MAX_MAPS];
};

template <typename T> __host__ __device__ constexpr size_t fl_z_bytes(const fft::Axis &ax, int pairs) {
    return ((size_t)ax.tw_len + (size_t)2 * pairs * fft::row_len(ax)) * 2 * sizeof(T);
}
template <typename T> __host__ __device__ constexpr int fl_z_pairs(const fft::Axis &ax) {
    int L = 128 / sl_z_threads(ax);
    if (L < 1) L = 1;
    while (L > 1 && fl_z_bytes<T>(ax, L) > (size_t)SL_SMEM) L /= 2;
    return L;
}

template <typename T> __global__ void fl_table_kernel(const __grid_constant__ SlParams p, typename cplx<T>::type *table) {
    sl_twiddles<T>(p.ay, table + p.tab_y, threadIdx.x, blockDim.x);
    sl_twiddles<T>(p.az, table + p.tab_z, threadIdx.x, blockDim.x);
}

// ---- Z: two real rows in, two half spectra out -----------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(128, SlShape<T>::ZBLOCKS)
    fl_z_kernel(const __grid_constant__ SlParams p, const typename cplx<T>::type *table, const T *R,
                typename cplx<T>::type *W) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const SlMap &mp = p.maps[blockIdx.y];
    const fft::AxisUse<N, true> use(p.az);
    const fft::Axis &az = use.v;
    const int nt = N ? sl_z_threads(az) : blockDim.x, L = N ? fl_z_pairs<T>(az) : blockDim.y, n = az.n, ld = fft::row_len(az);
    C *tw = reinterpret_cast<C *>(sl_smem), *sm = tw + az.tw_len + threadIdx.y * ld, *sm2 = sm + L * ld;
    C *res = az.np == 2 ? sm2 : sm;   // the buffer that the last pass does not read
    sl_load_table(tw, table + p.tab_z, az.tw_len);
    const int64_t pair = (int64_t)blockIdx.x * L + threadIdx.y, pairs = (int64_t)p.m0 * p.m1 / 2;
    const bool on = pair < pairs;
    const T *ra = R + ((int64_t)blockIdx.y * pairs + (on ? pair : 0)) * 2 * n, *rb = ra + n;
    C *wa = W + mp.w_off + (on ? 2 * pair * mp.ldz : 0), *wb = wa + mp.ldz;
    const int K = mp.kz_max;
    __syncthreads();   // the table
    fft::line_fft<T, -1>(
        use, threadIdx.x, nt, on, sm, sm2, tw, [&](int e) { return fft::row_at(az, e); },
        [&](int e, int) {
            C v;
            v.x = ra[e];
            v.y = rb[e];
            return v;
        },
        [&](int e, C v, int side) {
            const int kz = (side ? side > 0 : 2 * e > n) ? n - e : e;
            if (kz <= K) res[fft::row_at(az, e)] = v;
        });
    __syncthreads();
    if (!on) return;
    for (int kz = threadIdx.x; kz <= K; kz += nt) {
        const C f = res[fft::row_at(az, kz)], h = res[fft::row_at(az, kz ? n - kz : 0)];
        C a, b;
        a.x = (T)0.5 * (f.x + h.x);
        a.y = (T)0.5 * (f.y - h.y);
        b.x = (T)0.5 * (f.y + h.y);
        b.y = (T)0.5 * (h.x - f.x);
        wa[kz] = a;
        wb[kz] = b;
    }
}

// ---- Y: forward transform along y, in place ----------------------------------------------
template <typename T, int N>
__global__ void __launch_bounds__(SlShape<T>::THREADS, SlShape<T>::BLOCKS)
    fl_y_kernel(const __grid_constant__ SlParams p, const typename cplx<T>::type *table, typename cplx<T>::type *W) {
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
    __syncthreads();
    fft::line_fft<T, -1>(
        use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
        [&](int e, int) { return sl_elem(w, e, row); },
        [&](int e, C v, int side) {
            if (fft::abs_label(e, ay.n, side) <= ry) sl_elem(w, e, row) = v;
        });
}

// ---- X: forward transform along x, filter, sum over the maps of a shell -----------------------
// block (lines of kz, threads per line); grid (map-grid columns ky x runs, shells)
template <typename T, int N>
__global__ void __launch_bounds__(SlShape<T>::THREADS, SlShape<T>::BLOCKS)
    fl_x_kernel(const __grid_constant__ SlParams p, const __grid_constant__ FlShells sh, const typename cplx<T>::type *W,
                typename cplx<T>::type *grad) {
    using C = typename cplx<T>::type;
    extern __shared__ __align__(16) unsigned char sl_smem[];
    const Grid &g = p.g;
    const fft::AxisUse<N, true> use(p.ax);
    const fft::Axis &ax = use.v;
    const int L = N ? sl_lines<T>(ax) : blockDim.x, NT = N ? sl_threads<T>(ax) : blockDim.y, runs = p.kz_top / L + 1;
    const int run = blockIdx.x % runs, iy = blockIdx.x / runs, kz0 = run * L;
    const int ky = freq_index(iy, p.m1);                  // the band lies inside both grids
    double top = 0.0;
    for (int i = sh.first[blockIdx.y]; i < sh.first[blockIdx.y + 1]; ++i) top = fmax(top, p.maps[sh.order[i]].hi2);
    if (abs(ky) > sl_ky_radius(g, top, kz0)) return;      // (kz0 beyond every band: radius -1)
    C *tw = reinterpret_cast<C *>(sl_smem), *sm = tw + ax.tw_len, *sm2 = sm + ax.n * L;
    sl_twiddles<T>(ax, tw, threadIdx.y * blockDim.x + threadIdx.x, blockDim.x * blockDim.y);
    __syncthreads();
    const int line = threadIdx.x, kz = kz0 + line;
    const double kyv = __dmul_rn((double)ky, g.kf1), kzv = __dmul_rn((double)kz, g.kf2);
    const double ky2 = __dmul_rn(kyv, kyv), kz2 = __dmul_rn(kzv, kzv);
    const int64_t col = (int64_t)(ky < 0 ? ky + g.n1 : ky) * g.nh2 + kz, xstep = (int64_t)g.n1 * g.nh2;
    for (int i = sh.first[blockIdx.y]; i < sh.first[blockIdx.y + 1]; ++i) {
        const SlMap &mp = p.maps[sh.order[i]];
        if (kz0 > mp.kz_max || abs(ky) > sl_ky_radius(g, mp.hi2, kz0)) continue;   // the same for the whole block
        const bool on = kz <= mp.kz_max;
        const int r_out = sl_radius(mp.hi2, ky2 + kz2, g.kf0), r_in = sl_radius(mp.lo2, ky2 + kz2, g.kf0) - 2;
        const int wx = p.m1 * mp.ldz * (int)sizeof(C);
        const C *w = W + mp.w_off + (int64_t)iy * mp.ldz + kz;
        C *o = grad + mp.src * p.src_stride + col;
        fft::line_fft<T, -1>(
            use, threadIdx.y, NT, on, sm, sm2, tw, [&](int e) { return e * L + line; },
            [&](int e, int) { return sl_elem(w, e, wx); },
            [&](int e, C v, int side) {
                const int ka = fft::abs_label(e, ax.n, side);
                if (ka > r_out || ka < r_in) return;
                const int kx = (side ? side > 0 : e >= (ax.n >> 1)) ? -ka : ka;
                const double kxv = __dmul_rn((double)kx, g.kf0);
                const double s = __dadd_rn(__dadd_rn(__dmul_rn(kxv, kxv), ky2), kz2);
                if (!(mp.lo <= s && s < mp.hi)) return;
                double f = mp.scale;
                if (mp.l1) {
                    const double k = __dsqrt_rn(s);
                    f *= legendre(mp.l1, k != 0.0 ? __ddiv_rn(k_dot_los(g.los, g.l0, g.l1, g.l2, kxv, kyv, kzv), k) : 0.0);
                }
                C &q = o[(kx < 0 ? kx + g.n0 : kx) * xstep];
                q.x += (T)((double)v.x * f);
                q.y += (T)((double)v.y * f);
            });
        __syncthreads();   // the exchange buffers are free for the next map
    }
}

// ---- launches -------------------------------------------------------------------------------
enum FlStage { FL_Z, FL_Y, FL_X };

// one pass with the kernels of length N (0: the run-time plan); a.src: the real maps, a.out: the gradient
template <typename T, int N>
cudaError_t fl_launch(FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s) {
    using C = typename cplx<T>::type;
    cudaError_t e;
    if (stage == FL_Z) {
        const int t = sl_z_threads(p.az), L = fl_z_pairs<T>(p.az);
        const size_t smem = fl_z_bytes<T>(p.az, L);
        if ((e = sl_allow(fl_z_kernel<T, N>, smem)) != cudaSuccess) return e;
        const int64_t pairs = (int64_t)p.m0 * p.m1 / 2;
        fl_z_kernel<T, N><<<dim3((unsigned)((pairs + L - 1) / L), a.n_maps), dim3(t, L), smem, s>>>(
            p, (const C *)a.table, (const T *)a.src, (C *)a.W);
        return cudaGetLastError();
    }
    const fft::Axis &ax = stage == FL_X ? p.ax : p.ay;
    const int L = sl_lines<T>(ax), t = sl_threads<T>(ax), runs = p.kz_top / L + 1;
    const size_t smem = sl_line_bytes<T>(ax, L);
    if (stage == FL_Y) {
        if ((e = sl_allow(fl_y_kernel<T, N>, smem)) != cudaSuccess) return e;
        fl_y_kernel<T, N><<<dim3((unsigned)(p.m0 * runs), a.n_maps), dim3(L, t), smem, s>>>(p, (const C *)a.table, (C *)a.W);
    } else {
        if ((e = sl_allow(fl_x_kernel<T, N>, smem)) != cudaSuccess) return e;
        fl_x_kernel<T, N><<<dim3((unsigned)(p.m1 * runs), sh.n), dim3(L, t), smem, s>>>(p, sh, (const C *)a.W, (C *)a.out);
    }
    return cudaGetLastError();
}

// the lengths of SL_GROUP_* have kernels of their own
#define FL_CASE(N)                                                                                     \
    case N: *e = f64 ? fl_launch<double, N>(stage, p, sh, a, s) : fl_launch<float, N>(stage, p, sh, a, s); return true;
#define FL_ARGS int n, bool f64, FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s, cudaError_t *e
#define FL_DEFINE_GROUP(K)               \
    bool fl_group_##K(FL_ARGS) {         \
        switch (n) { SL_GROUP_##K(FL_CASE) } \
        return false;                    \
    }
cudaError_t fl_any_f64(FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s);
cudaError_t fl_any_f32(FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s);
bool fl_group_0(FL_ARGS);
bool fl_group_1(FL_ARGS);
bool fl_group_2(FL_ARGS);
bool fl_group_3(FL_ARGS);

}  // namespace pb
