// Host side of the band-limited chains (kernels and their description in pb_masked.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include "pb_masked.cuh"

namespace pb {
namespace fft {

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

struct MrLayout {
    Axis ax, ay, azi, azf;
    int tw_x, tw_y, tw_zi, tw_zf, tw_len;
};

static int mr_layout(const Grid &G, MrLayout *L) {
    // the larger radix where the operands come from memory: all of a thread's loads in one round
    L->ax = fft::make_axis(G.n0, true);
    L->ay = fft::make_axis(G.n1, true);
    L->azi = fft::make_axis(G.n2, false);
    L->azf = fft::make_axis(G.n2, true);
    if (!L->ax.np || !L->ay.np || !L->azi.np || std::max(G.n0, std::max(G.n1, G.n2)) > 1024)
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
    sh->Lx = line_count(p.ax);
    sh->Tx = line_threads(p.ax);
    sh->sx = line_bytes(p.ax, sh->Lx);
    sh->Ly = line_count(p.ay);
    sh->Ty = line_threads(p.ay);
    sh->sy = line_bytes(p.ay, sh->Ly);
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
    // every stage of a full chunk over all planes and rows can be launched
    p.n_x = G.n0;
    p.n_pairs = G.n0 * ((G.n1 + 1) / 2);
    for (MrStage stage : {MR_X, MR_Y, MR_Z, MR_PRODUCT, MR_Y_BACK, MR_X_BACK}) {
        const MrGrid n = mr_grid(stage, p, *sh, MR_MAX_MAPS);
        if (n.x > 2147483647 || n.y > 65535 || n.z > 65535) return fail(PB_ERR_UNSUPPORTED, "pb_masked_rows: too many rows");
    }
    return PB_OK;
}

// one stage of the maps in flight, with the kernels of length n where there are any
static int mr_stage(int n, MrStage stage, const MrParams &p, const MrShapes &sh, const MrArgs &a, cudaStream_t s,
                    const char *where) {
    cudaError_t e = cudaSuccess;
    if (!mr_group_0(n, stage, p, sh, a, s, &e) && !mr_group_1(n, stage, p, sh, a, s, &e) &&
        !mr_group_2(n, stage, p, sh, a, s, &e) && !mr_group_3(n, stage, p, sh, a, s, &e))
        e = mr_launch<0>(stage, p, sh, a, s);
    return e == cudaSuccess ? PB_OK : cuda_check(e, where);
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
    MrParams p;
    MrShapes sh;
    st = mr_setup(G, G.kf2 * G.nh2, &p, &sh);  // what has a table is taken whatever the band
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
    cudaStream_t s = as_stream(stream);
    MrArgs a{};
    a.src = (const double2 *)src;
    a.table = (const double2 *)table;
    a.mask = mask;
    a.pairs = pairs;
    a.xs = xs;
    a.x_on = x_on;
    a.pair_on = pair_on;
    a.W = (double2 *)workspace;
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
        a.maps = nm;
        a.out = (double2 *)out + (int64_t)m0 * G.nhalf;
        if ((st = mr_stage(G.n0, MR_X, p, sh, a, s, "pb_masked_rows(x)"))) return st;
        if ((st = mr_stage(G.n1, MR_Y, p, sh, a, s, "pb_masked_rows(y)"))) return st;
        if ((st = mr_stage(G.n2, MR_Z, p, sh, a, s, "pb_masked_rows(z)"))) return st;
        if ((st = mr_stage(G.n1, MR_Y_BACK, p, sh, a, s, "pb_masked_rows(y')"))) return st;
        if ((st = mr_stage(G.n0, MR_X_BACK, p, sh, a, s, "pb_masked_rows(x')"))) return st;
    }
    return PB_OK;
}

extern "C" int pb_product_rows(const pb_grid_t *g, const double *X, const double *Y, const double *Z,
                               const int32_t *pairs, int n_pairs, double k_out, const void *table, void *out,
                               void *workspace, size_t workspace_bytes, void *stream) {
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
    cudaStream_t s = as_stream(stream);
    MrArgs a{};
    a.X = X;
    a.Y = Y ? Y : X;
    a.Z = Z;
    a.table = (const double2 *)table;
    a.W = (double2 *)workspace;
    for (int m0 = 0; m0 < n_pairs; m0 += chunk) {
        a.maps = std::min(chunk, n_pairs - m0);
        for (int m = 0; m < a.maps; ++m) {
            a.products.i[m] = (int16_t)pairs[2 * (m0 + m)];
            a.products.j[m] = (int16_t)pairs[2 * (m0 + m) + 1];
        }
        a.out = (double2 *)out + (int64_t)m0 * G.nhalf;
        if ((st = mr_stage(G.n2, MR_PRODUCT, p, sh, a, s, "pb_product_rows(z)"))) return st;
        if ((st = mr_stage(G.n1, MR_Y_BACK, p, sh, a, s, "pb_product_rows(y)"))) return st;
        if ((st = mr_stage(G.n0, MR_X_BACK, p, sh, a, s, "pb_product_rows(x)"))) return st;
    }
    return PB_OK;
}
