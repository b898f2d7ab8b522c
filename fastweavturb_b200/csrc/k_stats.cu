// k_stats.cu -- statistics of the woven field:
//   minmax_kernel      component ranges, bit-exact (order-preserving integer atomics)
//   pdf_kernel         REAL(4) bin search of subroutine.f90:22-34 from the bin size and the
//                      edges beside the guess, integer shared-memory histograms
//   sp_kernel          longitudinal increments at separations r, moments p = 1..pmax
//                      accumulated in FP64 (subroutine.f90:64-129); lines staged in shared
//                      memory so each velocity component is read from HBM once
//   field_wh_kernel    downsampled |omega| and omega.u (tube.f90:1055-1071)
#include "k_common.cuh"

#include <cmath>
#include <type_traits>

namespace fwt {

// Component ranges, exact in the field's precision: FP32 values through order-preserving 32-bit
// atomics, FP64 values through 64-bit ones (mm: two words of the value's width per component,
// component blockIdx.y).  Bound by HBM: 16-byte loads, four of them in flight per thread.
template <typename Real>
__global__ void __launch_bounds__(256) minmax_kernel(const Real *__restrict__ f, size_t n, void *__restrict__ mm)
{
    Real mn = (Real)3.4e38f, mx = (Real)-3.4e38f;
    if (sizeof(Real) == 8) {
        mn = (Real)1.7e308;
        mx = (Real)-1.7e308;
    }
    constexpr int kV = 16 / sizeof(Real);
    struct __align__(16) Vec {
        Real v[kV];
    };
    const Real *a = f + blockIdx.y * n;   // n is a multiple of 8 (N is even): the components start on 16 bytes
    const size_t nv = n / kV, step = (size_t)gridDim.x * blockDim.x;
    const Vec *av = reinterpret_cast<const Vec *>(a);
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * step < nv; i += 4 * step) {
        Vec q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = av[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < kV; ++j) {
                mn = fmin(mn, q[k].v[j]);
                mx = fmax(mx, q[k].v[j]);
            }
    }
    for (; i < nv; i += step) {
        const Vec q = av[i];
#pragma unroll
        for (int j = 0; j < kV; ++j) {
            mn = fmin(mn, q.v[j]);
            mx = fmax(mx, q.v[j]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if constexpr (sizeof(Real) == 8) {
            unsigned long long *m = (unsigned long long *)mm + 2 * blockIdx.y;
            atomicMin(m, d2ord((double)mn));
            atomicMax(m + 1, d2ord((double)mx));
        } else {
            uint32_t *m = (uint32_t *)mm + 2 * blockIdx.y;
            atomicMin(m, f2ord((float)mn));
            atomicMax(m + 1, f2ord((float)mx));
        }
    }
}

// Histogram of v = (float)((double)x * s) over n values: bin = first l with v < hi[l], counted if
// lo[l] <= v.  The upper edges never decrease, so the bin is found from the guess (v - vmin) /
// bin size and the edges beside it, instead of a binary search (eight dependent shared loads at
// 201 bins).  The counts are kept in `copies` (a power of two up to 32) interleaved copies, lane
// i in copy i mod copies: with 32 every lane has its own bank and a field whose values crowd into
// one bin (omega between the tubes) costs no more than a flat one.  Six components of 512^3, 201
// bins: 4.96 ms with the search and one copy, 1.75 now; reading them takes 0.5.
template <typename Real>
__global__ void __launch_bounds__(256) pdf_kernel(const Real *__restrict__ a, size_t n, double s, float vmin, float ibsz,
                                                  const float *__restrict__ lo, const float *__restrict__ hi, int nbins,
                                                  int copies, unsigned long long *__restrict__ counts)
{
    extern __shared__ unsigned char smem[];
    float *s_hi = (float *)smem;
    float *s_lo = s_hi + nbins;
    uint32_t *s_cnt = (uint32_t *)(s_lo + nbins);
#pragma unroll 8
    for (int i = threadIdx.x; i < nbins; i += 256) {
        s_hi[i] = hi[i];
        s_lo[i] = lo[i];
    }
#pragma unroll 8
    for (int i = threadIdx.x; i < nbins * copies; i += 256) s_cnt[i] = 0;
    __syncthreads();
    const int mine = (int)threadIdx.x & (copies - 1);
    const float last = s_hi[nbins - 1];
    auto count = [&](Real x) {
        const float v = (float)((double)x * s);
        if (!(v < last)) return;   // beyond the last edge, or not a number
        int l = min(max((int)((v - vmin) * ibsz), 0), nbins - 1);
        while (l > 0 && v < s_hi[l - 1]) --l;
        while (!(v < s_hi[l])) ++l;
        if (s_lo[l] <= v) atomicAdd(s_cnt + l * copies + mine, 1u);
    };
    constexpr int kV = 16 / sizeof(Real);
    struct __align__(16) Vec {
        Real v[kV];
    };
    const size_t nv = n / kV, step = (size_t)gridDim.x * blockDim.x;   // n is a multiple of 8 (N is even)
    const Vec *av = reinterpret_cast<const Vec *>(a);
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (step >= n) {   // a small grid: one value a thread, over as many blocks as that gives
        if (i < n) count(a[i]);
        i = nv;
    }
    for (; i + step < nv; i += 2 * step) {
        const Vec p = av[i], q = av[i + step];
#pragma unroll
        for (int j = 0; j < kV; ++j) count(p.v[j]);
#pragma unroll
        for (int j = 0; j < kV; ++j) count(q.v[j]);
    }
    if (i < nv) {
        const Vec p = av[i];
#pragma unroll
        for (int j = 0; j < kV; ++j) count(p.v[j]);
    }
    __syncthreads();
    if (copies == 1) {
#pragma unroll 4
        for (int i2 = threadIdx.x; i2 < nbins; i2 += 256)
            if (s_cnt[i2]) atomicAdd(counts + i2, (unsigned long long)s_cnt[i2]);
        return;
    }
    for (int i2 = threadIdx.x; i2 < nbins; i2 += blockDim.x) {
        unsigned long long t = 0;
        for (int k = 0; k < copies; ++k) t += s_cnt[i2 * copies + ((k + i2) & (copies - 1))];
        if (t) atomicAdd(counts + i2, t);
    }
}

// Structure functions along one axis.  A block stages W lines of length N in shared memory
// as [pos][line] (padded), in the field's own precision; groups at the end of an axis may hold
// fewer lines, so any N works.  axis 0: u_x along x; 1: u_y along y; 2: u_z along z.
//
// Bound by FP64 arithmetic (the sums of du^p, p = 1..PMAX, over every point and separation) and by the
// staging of the lines, which nothing overlaps.  A warp takes up to four separations and a share of the
// positions, so a point is read and widened once for four increments; the sums use the even powers and
// fused multiply-adds (8 FP64 operations for p <= 6, 14 for 10, where a running power took 21), the scale
// s = 1/u' enters as the power of two just above it, exactly, when the lines are staged, and as the
// remainder in [0.5, 1) at the end, only as many orders as asked for are summed, and separations equal
// modulo N once (the host's list).  512^3, three components, orders 1-6: 14.5 ms with the running power to
// order 10, 6.8 now; at the FP64 rate the 17 separations take 3.8.
template <typename Real>
__host__ __device__ constexpr int sp_lines(int N)
{
    return N < (sizeof(Real) == 8 ? 16 : 32) ? N : (sizeof(Real) == 8 ? 16 : 32);
}
constexpr int kSpPerWarp = 4;   // separations of a warp at the most
static_assert(kSpPerWarp == 4, "sp_kernel's loops");
// Groups of separations in a block, and its threads.  The groups are spread evenly over as few blocks as
// hold them, and so are the separations over the groups; few groups share the positions among several
// warps each.  When a block took eight groups of four whether asked for or not, two warps to a group at
// the most, few separations took longer than with one warp each: 512^3, ms, so / now (one warp each): one
// separation, orders 1-6: 7.9 / 1.7 (5.3); 33, orders 1-10: 34.3 / 21.2 (28.7); 17, orders 1-6: 7.8 / 6.8
// (13.6).
constexpr int kSpGroups = 8, kSpMaxThreads = 384;
constexpr int kSpPositions = 16;   // positions a lane at the least, where positions are shared

template <int PMAX>
__device__ __forceinline__ void sp_accumulate(double d, double (&acc)[PMAX])
{
    const double d2 = d * d;
    acc[0] += d;
    acc[1] += d2;
    if (PMAX > 2) acc[2 < PMAX ? 2 : 0] = fma(d2, d, acc[2 < PMAX ? 2 : 0]);
    if (PMAX > 3) {
        const double d4 = d2 * d2;
        acc[3 < PMAX ? 3 : 0] += d4;
        if (PMAX > 4) acc[4 < PMAX ? 4 : 0] = fma(d4, d, acc[4 < PMAX ? 4 : 0]);
        if (PMAX > 5) {
            if (PMAX == 6) {
                acc[5 < PMAX ? 5 : 0] = fma(d4, d2, acc[5 < PMAX ? 5 : 0]);
            } else {
                const double d6 = d4 * d2, d8 = d4 * d4;
                acc[5 < PMAX ? 5 : 0] += d6;
                acc[6 < PMAX ? 6 : 0] = fma(d6, d, acc[6 < PMAX ? 6 : 0]);
                acc[7 < PMAX ? 7 : 0] += d8;
                acc[8 < PMAX ? 8 : 0] = fma(d8, d, acc[8 < PMAX ? 8 : 0]);
                acc[9 < PMAX ? 9 : 0] = fma(d8, d2, acc[9 < PMAX ? 9 : 0]);
            }
        }
    }
}

// The field is a box n0 x n1 x n2 (x fastest) whose extent along the axis is the line length N:
// the whole grid, or a z-slab (axes 0, 1) or y-pencil (axis 2) of a grid split over GPUs.  The
// axis is axis0 + blockIdx.y, its component stride elements further on per step.  blockDim is
// 32 x (groups of separations) x (shares of the positions); blockIdx.z takes the next groups.
// Scaled: each increment is multiplied by `post` in FP64, for a scale that says nothing about the
// field's size (a caller's own, or one beyond the staged type's exponents), where sc is 1.
template <typename Real, int PMAX, bool Scaled = false>
__global__ void __launch_bounds__(kSpMaxThreads, PMAX > 6 ? 1 : 2) sp_kernel(const Real *__restrict__ u0, size_t stride, int N, int n0, int n1, int n2,
                                                 int axis0, Real sc, double post, const int *__restrict__ rs,
                                                 int nr, int ngroups, double *__restrict__ Sp)
{
    extern __shared__ __align__(16) unsigned char sp_smem[];
    Real *tile = reinterpret_cast<Real *>(sp_smem);   // N x (W + 1)
    const int axis = axis0 + blockIdx.y;
    const Real *__restrict__ u = u0 + blockIdx.y * stride;
    const int W = sp_lines<Real>(N);
    const int ld = W + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // group g of all takes separations g, g + all, ...: four at the most, and none one more than another
    const int all = ngroups * (int)gridDim.z, group = (int)blockIdx.z * ngroups + warp % ngroups;
    const int count = group < nr ? (nr - 1 - group) / all + 1 : 0;
    // a lane's line, and the share of the positions that its part of the warp and its warp take
    const int per = 32 / W, line = lane % W, sub = lane / W;
    const int first = (warp / ngroups) * per + sub, pstep = (nwarps / ngroups) * per;
    double acc[kSpPerWarp][PMAX];
    int rr[kSpPerWarp];
#pragma unroll
    for (int a = 0; a < kSpPerWarp; ++a) {
#pragma unroll
        for (int p = 0; p < PMAX; ++p) acc[a][p] = 0.0;
        rr[a] = a < count ? rs[group + a * all] : 0;
    }
    // axis 0: groups of W consecutive x-rows (row = y + n1 z); axes 1, 2: groups of W
    // consecutive x at fixed z (axis 1) or fixed y (axis 2)
    const int xgroups = (n0 + W - 1) / W;
    const int64_t nrows = (int64_t)n1 * n2;
    const int64_t ntiles = axis == 0 ? (nrows + W - 1) / W : (int64_t)xgroups * (axis == 1 ? n2 : n1);
    for (int64_t g = blockIdx.x; g < ntiles; g += gridDim.x) {
        __syncthreads();
        int nl;   // lines of this tile
        if (axis == 0) {
            const int64_t row0 = g * W;
            nl = (int)min((int64_t)W, nrows - row0);
            for (int l = warp; l < nl; l += nwarps)
                for (int x = lane; x < N; x += 32) tile[x * ld + l] = u[(size_t)(row0 + l) * n0 + x] * sc;
        } else {
            const int xg = (int)(g % xgroups), o = (int)(g / xgroups);
            const int x0 = xg * W;
            nl = min(W, n0 - x0);
            const size_t base = axis == 1 ? (size_t)n0 * ((size_t)n1 * o) : (size_t)n0 * o;
            const size_t ps = axis == 1 ? (size_t)n0 : (size_t)n0 * n1;
            if (line < nl && sub < per)
                for (int pos = warp * per + sub; pos < N; pos += nwarps * per)
                    tile[pos * ld + line] = u[base + ps * pos + x0 + line] * sc;
        }
        __syncthreads();
        if (line < nl && sub < per) {
            auto run = [&](auto n) {
                for (int pos = first; pos < N; pos += pstep) {
                    const double c = (double)tile[pos * ld + line];
#pragma unroll
                    for (int a = 0; a < decltype(n)::value; ++a) {
                        int q = pos + rr[a];
                        if (q >= N) q -= N;
                        const double d = (double)tile[q * ld + line] - c;
                        sp_accumulate<PMAX>(Scaled ? d * post : d, acc[a]);
                    }
                }
            };
            if (count == 4) run(std::integral_constant<int, 4>{});
            else if (count == 3) run(std::integral_constant<int, 3>{});
            else if (count == 2) run(std::integral_constant<int, 2>{});
            else if (count == 1) run(std::integral_constant<int, 1>{});
        }
    }
    // the shares' sums meet in shared memory, so that a block adds each sum once
    double *part = reinterpret_cast<double *>(sp_smem);   // [warp][separation of the group][order]
    __syncthreads();
#pragma unroll
    for (int a = 0; a < kSpPerWarp; ++a) {
        if (a >= count) break;
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            const double v = warp_sum(acc[a][p]);
            if (lane == 0) part[(warp * kSpPerWarp + a) * PMAX + p] = v;
        }
    }
    __syncthreads();
    const int per_group = kSpPerWarp * PMAX;
    for (int i = threadIdx.x; i < ngroups * per_group; i += blockDim.x) {
        const int m = (int)blockIdx.z * ngroups + i / per_group + i % per_group / PMAX * all;
        if (m >= nr) continue;
        double v = 0.0;
        for (int w = 0; w < nwarps; w += ngroups) v += part[w * per_group + i];
        atomicAdd(Sp + i % PMAX * nr + m, v);
    }
}

template <typename Real>
__global__ void field_wh_kernel(const Real *__restrict__ w, const Real *__restrict__ u, int N, int nd, double s,
                                float *__restrict__ out)
{
    const size_t n3 = (size_t)N * N * N;
    const int rd = N / nd;
    const size_t m3 = (size_t)nd * nd * nd;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < m3; q += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % nd), j = (int)((q / nd) % nd), k = (int)(q / ((size_t)nd * nd));
        // data_box(i, j, k) = field(i*r_d, j*r_d, k*r_d), 1-based
        const size_t g = (size_t)((i + 1) * rd - 1) + (size_t)N * ((size_t)((j + 1) * rd - 1) + (size_t)N * ((k + 1) * rd - 1));
        const double wx = (double)w[g] * s, wy = (double)w[g + n3] * s, wz = (double)w[g + 2 * n3] * s;
        const double ux = (double)u[g] * s, uy = (double)u[g + n3] * s, uz = (double)u[g + 2 * n3] * s;
        out[q] = (float)sqrt(wx * wx + wy * wy + wz * wz);
        out[q + m3] = (float)(wx * ux + wy * uy + wz * uz);
    }
}

__global__ void mm_init2(void *mm, int n, int wide)
{
    const int i = threadIdx.x;
    if (i >= n) return;
    if (wide) ((unsigned long long *)mm)[i] = (i & 1) ? 0ull : ~0ull;
    else ((uint32_t *)mm)[i] = (i & 1) ? 0u : 0xffffffffu;
}

static unsigned grid_for(Ctx *c, size_t n, int per_sm = 8)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->dev);
    return (unsigned)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, (size_t)sms * per_sm));
}

// raw component ranges of u (which = 1) or omega (which = 0), exact in the field's precision
int stats_minmax(Ctx *c, int which)
{
    const size_t n3 = field_elems(c);
    void *f = which ? c->b_u.p : c->b_w.p;
    const bool wide = c->p.precision == 64;
    FWT_TRY(buf_reserve(c, c->scratch[19], 128));
    char *mm = (char *)c->scratch[19].p + 16;
    const int km = kt_begin(c, KT_STATS);
    mm_init2<<<1, 32, 0, c->stream>>>(mm, 6, wide ? 1 : 0);
    const dim3 g(grid_for(c, n3 / (wide ? 2 : 4), 4), 3);
    if (wide) minmax_kernel<double><<<g, 256, 0, c->stream>>>((const double *)f, n3, mm);
    else minmax_kernel<float><<<g, 256, 0, c->stream>>>((const float *)f, n3, mm);
    kt_end(c, km);
    c->launches += 2;
    FWT_CUDA(cudaGetLastError());
    unsigned long long h[6];
    FWT_CUDA(cudaMemcpyAsync(h, mm, wide ? 48 : 24, cudaMemcpyDeviceToHost, c->stream));
    FWT_CUDA(cudaStreamSynchronize(c->stream));
    std::vector<double> &mn = which ? c->umin : c->wmin, &mx = which ? c->umax : c->wmax;
    mn.assign(3, 0.0);
    mx.assign(3, 0.0);
    const uint32_t *h32 = (const uint32_t *)h;
    for (int d = 0; d < 3; ++d) {
        mn[d] = wide ? ord2d(h[2 * d]) : (double)ord2f(h32[2 * d]);
        mx[d] = wide ? ord2d(h[2 * d + 1]) : (double)ord2f(h32[2 * d + 1]);
    }
    if (which) c->umm_valid = true;
    else c->wmm_valid = true;
    return 0;
}

int stats_normalise(Ctx *c)
{
    if (c->slab_nz) return fail(FWT_E_STATE, "normalise: not available on a z-slab context");
    if (!c->have_u) return fail(FWT_E_STATE, "normalise before Biot-Savart");
    // Etot = sum u.u dv / 2 / (2pi)^3 = 1/2 <u^2>; up = sqrt(2 Etot / 3) (tube.f90:1028-1030)
    c->Etot = c->Etot_raw;
    c->up = std::sqrt(2 * c->Etot / 3);
    c->enstrophy = c->enstrophy_raw / (c->up * c->up);
    c->normalised = true;
    return 0;
}

// host-side REAL(4) bin layout, identical to the reference's (subroutine.f90:12-20)
static void pdf_layout(float vmin, float vmax, int nbins, std::vector<float> &val, std::vector<float> &lo,
                       std::vector<float> &hi, float &bsz)
{
    bsz = (float)((float)(vmax - vmin) / (float)nbins);
    val.resize(nbins);
    lo.resize(nbins);
    hi.resize(nbins);
    const float half = (float)(0.5f * bsz);
    for (int l = 0; l < nbins; ++l) {
        const float prod = (float)((float)l * bsz);
        val[l] = (float)((double)vmin + 0.5 * (double)bsz + (double)prod);
        lo[l] = (float)(val[l] - half);
        hi[l] = (float)(val[l] + half);
    }
}

int stats_pdf(Ctx *c, int which, int comp, int nbins, float *val, float *pdf, uint64_t *counts)
{
    if (c->slab_nz) return fail(FWT_E_STATE, "pdf: not available on a z-slab context");
    if (which != 0 && which != 1) return fail(FWT_E_ARG, "pdf: which must be 0 (u) or 1 (omega)");
    if (comp < -1 || comp > 2) return fail(FWT_E_ARG, "pdf: component must be -1..2");
    if (nbins < 1 || nbins > 8192) return fail(FWT_E_ARG, "pdf: nbins must be 1..8192");
    if (!c->normalised) return fail(FWT_E_STATE, "pdf before normalisation");
    const bool is_u = which == 0;
    if (is_u && !c->umm_valid) FWT_TRY(stats_minmax(c, 1));
    if (!is_u && !c->wmm_valid) FWT_TRY(stats_minmax(c, 0));
    const std::vector<double> &mn = is_u ? c->umin : c->wmin, &mx = is_u ? c->umax : c->wmax;
    const double s = 1.0 / c->up;
    double rmin = 1.7e308, rmax = -1.7e308;
    for (int d = 0; d < 3; ++d) {
        if (comp >= 0 && d != comp) continue;
        rmin = std::min(rmin, mn[d]);
        rmax = std::max(rmax, mx[d]);
    }
    // range of the scaled REAL(4) values (float)(x s): rounding is monotone, so it is the
    // rounded scaled range of the exact raw values
    const float vmin = (float)(rmin * s), vmax = (float)(rmax * s);
    std::vector<float> hval, hlo, hhi;
    float bsz;
    pdf_layout(vmin, vmax, nbins, hval, hlo, hhi, bsz);
    FWT_TRY(buf_reserve(c, c->scratch[10], sizeof(float) * 2 * nbins + sizeof(unsigned long long) * nbins + 64));
    float *d_lo = (float *)c->scratch[10].p, *d_hi = d_lo + nbins;
    unsigned long long *d_cnt = (unsigned long long *)(((uintptr_t)(d_hi + nbins) + 15) & ~(uintptr_t)15);
    FWT_CUDA(cudaMemcpyAsync(d_lo, hlo.data(), sizeof(float) * nbins, cudaMemcpyHostToDevice, c->stream));
    FWT_CUDA(cudaMemcpyAsync(d_hi, hhi.data(), sizeof(float) * nbins, cudaMemcpyHostToDevice, c->stream));
    FWT_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(unsigned long long) * nbins, c->stream));
    const size_t n3 = field_elems(c);
    const void *f = is_u ? c->b_u.p : c->b_w.p;
    // the components lie one after the other: one launch takes one of them or all three
    const size_t o = comp < 0 ? 0 : (size_t)comp * n3, nv = comp < 0 ? 3 * n3 : n3;
    unsigned grid = grid_for(c, nv, 4);   // a value a thread, where the chip holds as many
    if ((size_t)grid * 256 < nv) grid = grid_for(c, nv / (c->p.precision == 64 ? 2 : 4), 4);
    // copies of the counts: as many as fit 40 KB beside the edges, up to one per lane, and no more counts
    // than a block has values (one component of 32^3, 200 bins, the whole call: 48 us with 16 copies and four
    // values a thread, 42 so)
    int copies = 1;
    while (copies < 32 && sizeof(float) * nbins * (2 + 2 * (size_t)copies) <= 40960 &&
           (size_t)nbins * copies * 2 <= nv / grid)
        copies *= 2;
    const size_t shb = sizeof(float) * 2 * nbins + sizeof(uint32_t) * nbins * (size_t)copies;
    // 8192 bins take 96 KB of shared memory, above the default 48 KB: the limit is raised to
    // the device's opt-in maximum, the same value for every context (the attribute belongs to
    // the kernel, for the whole process)
    int optin = 0;
    FWT_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->dev));
    if (shb > (size_t)optin) return fail(FWT_E_RANGE, "pdf: bins exceed one block's shared memory");
    if (c->p.precision == 64)
        FWT_CUDA(cudaFuncSetAttribute(pdf_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    else
        FWT_CUDA(cudaFuncSetAttribute(pdf_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    const int km = kt_begin(c, KT_STATS);
    const float ibsz = bsz > 0.0f ? 1.0f / bsz : 0.0f;
    if (c->p.precision == 64)
        pdf_kernel<double><<<grid, 256, shb, c->stream>>>((const double *)f + o, nv, s, vmin, ibsz, d_lo,
                                                                            d_hi, nbins, copies, d_cnt);
    else
        pdf_kernel<float><<<grid, 256, shb, c->stream>>>((const float *)f + o, nv, s, vmin, ibsz, d_lo,
                                                                           d_hi, nbins, copies, d_cnt);
    c->launches += 1;
    kt_end(c, km);
    FWT_CUDA(cudaGetLastError());
    std::vector<unsigned long long> hc(nbins);
    FWT_CUDA(cudaMemcpyAsync(hc.data(), d_cnt, sizeof(unsigned long long) * nbins, cudaMemcpyDeviceToHost, c->stream));
    FWT_CUDA(cudaStreamSynchronize(c->stream));
    // pdf_v(l)/(bin_size*nx*ny*nzp*nproc), left to right in REAL(4) (subroutine.f90:38)
    const int N = c->p.N;
    const int nz_eff = comp < 0 ? 3 * N : N;
    float den = bsz;
    den = (float)(den * (float)N);
    den = (float)(den * (float)N);
    den = (float)(den * (float)nz_eff);
    for (int l = 0; l < nbins; ++l) {
        if (val) val[l] = hval[l];
        if (pdf) pdf[l] = (float)((float)hc[l] / den);
        if (counts) counts[l] = hc[l];
    }
    return 0;
}

// Sums of du^p, p = 1..pmax, on a box (n0 x n1 x n2) of `axes` consecutive axes from axis0 (one
// component each, `stride` elements apart): sums[(p - 1) * nr + m] = sum (du s)^p at separation
// r[m].  Separations equal modulo N are summed once.  own_scale: s is 1/u' of this very field, so that
// u s is of order one.
static int sp_sums(Ctx *c, const void *u, size_t stride, int n0, int n1, int n2, int axis0, int axes, double s,
                   bool own_scale, int pmax, const int *r, int nr, double *sums)
{
    const int N = c->p.N;
    const bool f64 = c->p.precision == 64;
    const int W = f64 ? sp_lines<double>(N) : sp_lines<float>(N);
    // the staged lines, and in their place at the end the warps' sums
    const size_t shb = std::max((f64 ? sizeof(double) : sizeof(float)) * (size_t)N * (W + 1),
                                sizeof(double) * (kSpMaxThreads / 32) * kSpPerWarp * 10);
    // The dynamic shared-memory limit is a property of the kernel for the whole process: every
    // context sets the same value, the device's opt-in maximum, so that contexts of different N
    // on concurrent host threads never lower it under another's launch.
    int optin = 0;
    FWT_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->dev));
    if (shb > (size_t)optin) return fail(FWT_E_RANGE, "Sp: N too large for one block's shared memory");
    std::vector<int> uniq, at(nr);
    for (int m = 0; m < nr; ++m) {
        const int q = r[m] % N;
        size_t i = 0;
        while (i < uniq.size() && uniq[i] != q) ++i;
        if (i == uniq.size()) uniq.push_back(q);
        at[m] = (int)i;
    }
    // the power of two just above s scales the staged lines exactly; the rest, in [0.5, 1), is applied
    // below.  Any other scale (zero, negative, not finite, or beyond the staged type's exponents) and a
    // scale that need not fit the field, whose product with it could leave that type's range, multiplies
    // each increment in FP64 instead
    int e = 0;
    std::frexp(s, &e);
    const int emax = f64 ? 1000 : 120;
    const bool staged = own_scale && std::isfinite(s) && s > 0 && e > -emax && e < emax;
    const double sc = staged ? std::ldexp(1.0, e) : 1.0;
    const int P = !staged ? 10 : (pmax <= 4 ? 4 : (pmax <= 6 ? 6 : 10)), nu = (int)uniq.size();
    std::vector<double> h((size_t)P * nu);
    FWT_TRY(buf_reserve(c, c->scratch[9], sizeof(int) * 64 + sizeof(double) * 10 * 64 + 64));
    int *d_r = (int *)c->scratch[9].p;
    double *d_sp = (double *)((char *)c->scratch[9].p + 256);
    FWT_CUDA(cudaMemcpyAsync(d_r, uniq.data(), sizeof(int) * nu, cudaMemcpyHostToDevice, c->stream));
    FWT_CUDA(cudaMemsetAsync(d_sp, 0, sizeof(double) * P * nu, c->stream));
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->dev);
    const int64_t tiles = (int64_t)n0 * n1 * n2 / N / W + 1;
    const int all = (nu + kSpPerWarp - 1) / kSpPerWarp, nz = (all + kSpGroups - 1) / kSpGroups;
    const int ngroups = (all + nz - 1) / nz;
    const int shares = std::min(kSpMaxThreads / 32 / ngroups, std::max(1, N * W / 32 / kSpPositions));
    const unsigned threads = 32u * (unsigned)(ngroups * shares);
    const dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sms * 2)), (unsigned)axes, (unsigned)nz);
    const int km = kt_begin(c, KT_STATS);
#define FWT_SP(REAL, ...)                                                                                          \
do {                                                                                                           \
    auto k = sp_kernel<REAL, __VA_ARGS__>;                                                                     \
    FWT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));                    \
    k<<<grid, threads, shb, c->stream>>>((const REAL *)u, stride, N, n0, n1, n2, axis0, (REAL)sc, s, d_r, nu, ngroups, d_sp); \
} while (0)
    if (f64) {
        if (!staged) FWT_SP(double, 10, true); else if (P == 4) FWT_SP(double, 4);
        else if (P == 6) FWT_SP(double, 6); else FWT_SP(double, 10);
    } else {
        if (!staged) FWT_SP(float, 10, true); else if (P == 4) FWT_SP(float, 4);
        else if (P == 6) FWT_SP(float, 6); else FWT_SP(float, 10);
    }
#undef FWT_SP
    kt_end(c, km);
    c->launches += 1;
    FWT_CUDA(cudaGetLastError());
    FWT_CUDA(cudaMemcpyAsync(h.data(), d_sp, sizeof(double) * P * nu, cudaMemcpyDeviceToHost, c->stream));
    FWT_CUDA(cudaStreamSynchronize(c->stream));
    double f = 1.0;
    for (int p = 0; p < pmax; ++p) {
        f *= staged ? s / sc : 1.0;
        for (int m = 0; m < nr; ++m) sums[p * nr + m] = h[(size_t)p * nu + at[m]] * f;
    }
    return 0;
}

int stats_sp(Ctx *c, int pmax, const int *r, int nr, double *Sp)
{
    if (c->slab_nz) return fail(FWT_E_STATE, "S_p: not available on a z-slab context");
    if (!c->normalised) return fail(FWT_E_STATE, "structure functions before normalisation");
    if (pmax < 1 || pmax > 10) return fail(FWT_E_ARG, "Sp: pmax must be 1..10");
    if (nr < 1 || nr > 64) return fail(FWT_E_ARG, "Sp: nr must be 1..64");
    const int N = c->p.N;
    for (int m = 0; m < nr; ++m)
        if (r[m] < 0) return fail(FWT_E_ARG, "Sp: negative separation");
    FWT_TRY(sp_sums(c, c->b_u.p, field_elems(c), N, N, N, 0, 3, 1.0 / c->up, true, pmax, r, nr, Sp));
    const double inv = 1.0 / ((double)N * N * N * 3.0);
    for (int i = 0; i < pmax * nr; ++i) Sp[i] *= inv;
    return 0;
}

int stats_field_wh(Ctx *c, float *host_out)
{
    if (c->slab_nz) return fail(FWT_E_STATE, "field output: not available on a z-slab context");
    if (!c->normalised) return fail(FWT_E_STATE, "field output before normalisation");
    const int N = c->p.N, nd = c->p.N_downsample;
    if (nd < 1 || N % nd) return fail(FWT_E_ARG, "N_downsample must divide N");
    const size_t m3 = (size_t)nd * nd * nd, n3 = field_elems(c);
    FWT_TRY(buf_reserve(c, c->scratch[8], sizeof(float) * 2 * m3));
    float *d = (float *)c->scratch[8].p;
    const double s = 1.0 / c->up;
    const int km = kt_begin(c, KT_STATS);
    if (c->p.precision == 64)
        field_wh_kernel<double><<<grid_for(c, m3), 256, 0, c->stream>>>((const double *)c->b_w.p,
                                                                        (const double *)c->b_u.p, N, nd, s, d);
    else
        field_wh_kernel<float><<<grid_for(c, m3), 256, 0, c->stream>>>((const float *)c->b_w.p, (const float *)c->b_u.p,
                                                                       N, nd, s, d);
    kt_end(c, km);
    c->launches += 1;
    FWT_CUDA(cudaGetLastError());
    (void)n3;
    if (host_out) {
        FWT_CUDA(cudaMemcpyAsync(host_out, d, sizeof(float) * 2 * m3, cudaMemcpyDeviceToHost, c->stream));
        FWT_CUDA(cudaStreamSynchronize(c->stream));
    }
    return 0;
}

int stats_copy_field(Ctx *c, int which, int comp, double *host)
{
    if (which != 0 && which != 1) return fail(FWT_E_ARG, "copy_field: which must be 0 (omega) or 1 (u)");
    if (comp < 0 || comp > 2) return fail(FWT_E_ARG, "copy_field: component must be 0..2");
    if (which == 0 && !c->have_w) return fail(FWT_E_STATE, "omega not built");
    if (which == 1 && !c->have_u) return fail(FWT_E_STATE, "u not built");
    const size_t n3 = field_elems(c);
    const double s = c->normalised ? 1.0 / c->up : 1.0;
    const void *f = which ? c->b_u.p : c->b_w.p;
    if (c->p.precision == 64) {
        FWT_CUDA(cudaMemcpyAsync(host, (const double *)f + comp * n3, sizeof(double) * n3, cudaMemcpyDeviceToHost,
                                 c->stream));
        FWT_CUDA(cudaStreamSynchronize(c->stream));
        if (s != 1.0)
            for (size_t i = 0; i < n3; ++i) host[i] = host[i] * s;
    } else {
        std::vector<float> tmp(n3);
        FWT_CUDA(cudaMemcpyAsync(tmp.data(), (const float *)f + comp * n3, sizeof(float) * n3, cudaMemcpyDeviceToHost,
                                 c->stream));
        FWT_CUDA(cudaStreamSynchronize(c->stream));
        for (size_t i = 0; i < n3; ++i) host[i] = (double)tmp[i] * s;
    }
    return 0;
}

// S_p sums of one velocity component on a box (a z-slab or y-pencil of a grid split over GPUs):
// sums[p * nr + m] = sum over the box's lines along `axis` of (du s)^(p+1), du the increment at
// separation r[m]; the line axis must span the grid (extent N).  Not normalised: the caller adds
// the three components' sums over all boxes and divides by 3 N^3, as stats_sp does.
int stats_sp_block(Ctx *c, const void *u, int n0, int n1, int n2, int axis, double s, const int *r, int nr,
                   double *sums)
{
    const int N = c->p.N;
    if (axis < 0 || axis > 2) return fail(FWT_E_ARG, "sp_block: axis must be 0..2");
    const int ext[3] = {n0, n1, n2};
    if (ext[axis] != N || n0 < 1 || n1 < 1 || n2 < 1) return fail(FWT_E_ARG, "sp_block: the line axis must span N");
    if (nr < 1 || nr > 64) return fail(FWT_E_ARG, "sp_block: nr must be 1..64");
    for (int m = 0; m < nr; ++m)
        if (r[m] < 0) return fail(FWT_E_ARG, "sp_block: negative separation");
    return sp_sums(c, u, 0, n0, n1, n2, axis, 1, s, false, 10, r, nr, sums);
}

}  // namespace fwt
