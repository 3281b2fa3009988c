// ga_hydro.cuh - the hydrostatic equation set (HYDROSTATIC): integrate_hydro
// (solver.cpp:33-80) advects u and v, solves for pressure with
// solve_hydrostatic_pressure (pressure.cpp:229-298) and applies the
// pressure-gradient force with the factor cp * tbv; w is diagnosed from the
// anelastic continuity equation after each stage (w_velocity_LH,
// solver.cpp:144-163) and lives in the current slot only.
//
// The pressure is a lid pressure plus the hydrostatic integral of the
// buoyancy.  The lid pressure solves a 2-D Poisson problem for the
// density-weighted column divergence (poisson_fft2d, pressure.cpp:652-715):
// a transform along x, scaled by 1/nx, one tridiagonal solve along y per
// x-wavenumber (whose back substitution leaves the last row at its
// transformed value), and the inverse transform.  The transforms reuse the
// shared-memory Stockham FFT of the 3-D solve (fft_smem), batched over a tile
// of y-lines; the tridiagonal solves run in the context's precision with
// elimination factors formed once on the host in FP64.  Non-periodic domains.
#pragma once
#include "ga_kernels.cuh"

namespace ga {

template <typename T>
struct HydArgs {
    const T *dzu, *dzw;    // DZU(k) = zsw[k+1]-zsw[k], DZW(k) = zsu[k]-zsu[k-1] (model.h:205-206)
    // the tridiagonal system of init_fft2d (pressure.cpp:621-641) does not
    // change during a run: its elimination factors P[j+1] = -ccoef[j]/denom
    // and 1/denom, denom = BCOEF(i,j) + acoef[j] P[j], are formed once on the
    // host (the reference's expressions, FP64, stored in the context's
    // precision: FP64 is scarce on this GPU, and the FP32 solve keeps the
    // FP32 step's accuracy), [ny+1][nx] and [ny][nx] (x-wavenumber fastest:
    // a warp of wavenumbers reads one row at a time)
    const T *pf, *rden;
    const T *ac;           // acoef [ny]
    T *tw;                 // work of the tridiagonal solves where shared memory is too small, or null
    T *div;                // div_avg, [nx][ny]
    typename V2<T>::t *spec2;  // transformed div_avg, [ny][nx]
    T rhoavg;              // column-average density (column_average_density, initializer.cpp:1265-1282)
    T dz;
};

// The column kernels below hold HC columns per block with their levels in
// shared memory, a warp per column at a time with lanes over the levels; the
// pointwise parts of each recurrence (and its level factors) are formed by all
// lanes, then one thread per column runs the bare recurrence in the
// reference's order from shared memory.
constexpr int HC = 16, HC_THREADS = 128, HC_WARPS = HC_THREADS / 32;

// columns, and three rows of level factors
template <typename T>
__host__ __device__ constexpr size_t hyd_col_smem(int nz)
{
    return (2 * (size_t)HC + 3) * nz * sizeof(T);
}

// the columns that take column (i, j)'s value: itself and the lateral edges
// that mirror it (mirror_boundaries, boundaries.cpp:331-379; a corner takes
// the diagonal neighbour, as the reference's two passes leave it)
template <typename F>
__device__ __forceinline__ void with_mirrors(int nx, int ny, int i, int j, F f)
{
    const int ie = i == 1 ? 0 : i == nx - 2 ? nx - 1 : i, je = j == 1 ? 0 : j == ny - 2 ? ny - 1 : j;
    f(i, j);
    if (ie != i) f(ie, j);
    if (je != j) f(i, je);
    if (ie != i && je != j) f(ie, je);
}

// density-weighted column divergence of the forecast u, v (pressure.cpp:248-261)
// with its lateral mirror copies
template <typename T>
__global__ void __launch_bounds__(HC_THREADS) k_hyd_divavg(KParams<T> p, KFields<T> F, HydArgs<T> h, T step)
{
    extern __shared__ unsigned char hyd_smem[];
    T *term = (T *)hyd_smem;  // [HC][nz]
    const int nyi = p.ny - 2, nz = p.nz, lane = threadIdx.x & 31;
    const int ncol = (p.nx - 2) * nyi, col0 = blockIdx.x * HC;
    const T *UP = F.P[FU], *VP = F.P[FV];
    const long sx = (long)p.ny * nz, sy = nz;
    for (int cl = threadIdx.x >> 5; cl < HC && col0 + cl < ncol; cl += HC_WARPS) {
        const int col = col0 + cl, ci = col / nyi;
        const long c0 = gix(p.ny, nz, 1 + ci, 1 + col - ci * nyi, 0);
        for (int k = 1 + lane; k < nz - 1; k += 32) {
            const long c = c0 + k;
            term[cl * nz + k] =
                p.rhou[k] * h.dzu[k] * ((UP[c + sx] - UP[c]) * p.one_d_dx + (VP[c + sy] - VP[c]) * p.one_d_dy);
        }
    }
    __syncthreads();
    const int col = col0 + threadIdx.x;
    if (threadIdx.x >= HC || col >= ncol) return;
    T d = T(0), zsum = T(0);
#pragma unroll 8
    for (int k = 1; k < nz - 1; k++) {
        d += term[threadIdx.x * nz + k];
        zsum += h.dzu[k];
    }
    d /= (T(1004) * zsum * step * p.dt);
    const int ci = col / nyi;
    with_mirrors(p.nx, p.ny, 1 + ci, 1 + col - ci * nyi, [&](int i, int j) { h.div[(long)i * p.ny + j] = d; });
}

// transform along x of L y-lines (block (L, any)): forward from div_avg with
// the 1/nx scaling, or inverse into div_avg (real part)
template <typename T>
__global__ void k_hyd_fft(KParams<T> p, HydArgs<T> h, FftPlan P, const typename V2<T>::t *tw, int inv, int L)
{
    typedef typename V2<T>::t T2;
    extern __shared__ unsigned char smem_raw[];
    T2 *a = (T2 *)smem_raw;
    T2 *b = a + (long)p.nx * L;
    const int j0 = blockIdx.x * L;
    const int lt = min(L, p.ny - j0);
    for (int i = threadIdx.y; i < p.nx; i += blockDim.y)
        for (int l = threadIdx.x; l < L; l += blockDim.x) {
            T2 v;
            if (l < lt) {
                if (inv) {
                    v = h.spec2[(long)(j0 + l) * p.nx + i];
                } else {
                    v.x = h.div[(long)i * p.ny + j0 + l];
                    v.y = T(0);
                }
            } else {
                v.x = T(0);
                v.y = T(0);
            }
            a[i * L + l] = v;
        }
    __syncthreads();
    const T2 *r = inv ? fft_smem<true, T, T2>(a, b, L, P, tw, L) : fft_smem<false, T, T2>(a, b, L, P, tw, L);
    const T n = (T)p.nx;
    for (int i = threadIdx.y; i < p.nx; i += blockDim.y)
        for (int l = threadIdx.x; l < lt; l += blockDim.x) {
            const T2 v = r[i * L + l];
            if (inv) {
                h.div[(long)i * p.ny + j0 + l] = v.x;
            } else {
                T2 o;
                o.x = v.x / n;
                o.y = v.y / n;
                h.spec2[(long)(j0 + l) * p.nx + i] = o;
            }
        }
}

// the tridiagonal solves along y of HT x-wavenumbers (pressure.cpp:675-700),
// real and imaginary parts, with the precomputed factors: each step of the
// recurrence is a multiply-subtract and a multiply by 1/denom (the reference
// divides by denom; the two differ by an ulp, well inside the transform's own
// rounding).  Rows are [j][i]: the block stages its wavenumbers' rows and
// factors into shared memory at once, then two threads a wavenumber (real and
// imaginary) run the bare chain of 2 NY steps from there.  With a thread per
// wavenumber reading its rows from L2 in chunks it took 22 us at 128x128 in
// FP32; now 8.
constexpr int HT = 4, HT_THREADS = 128;
template <typename T>
__host__ __device__ constexpr size_t hyd_thomas_smem(int ny)
{
    return (size_t)HT * ny * 4 * sizeof(T);
}
// v: [j][HT] (re, im), the rows, then Q, then the solution
template <typename T>
__device__ __forceinline__ void hyd_thomas_body(const KParams<T> &p, const HydArgs<T> &h, T *v)
{
    typedef typename V2<T>::t T2;
    const int nj = p.ny, nx = p.nx, i0 = blockIdx.x * HT, nt = min(HT, nx - i0);
    T *r = v + (size_t)2 * HT * nj;             // [j][HT]: 1/denom
    T *pf = r + (size_t)HT * nj;                // [j][HT]: P[j+1]
    for (int w = threadIdx.x; w < HT * nj; w += HT_THREADS) {
        const int j = w / HT, t = min(w % HT, nt - 1);
        const long g = (long)j * nx + i0 + t;
        const T2 x = h.spec2[g];
        v[2 * w] = x.x;
        v[2 * w + 1] = x.y;
        r[w] = h.rden[g];
        pf[w] = h.pf[g + nx];
    }
    __syncthreads();
    if (threadIdx.x < 2 * HT) {
        // chunks of rows are read before their steps run, so a chunk waits on
        // shared memory once
        constexpr int CH = 8;
        const int t = threadIdx.x >> 1;
        T *c = v + threadIdx.x;
        const T last = c[2 * HT * (nj - 1)];  // the last row keeps its transformed value
        const T a1 = h.ac[1];                 // acoef: 0 in row 0, 1/dy^2 above
        T q = T(0);
        for (int j0 = 0; j0 < nj; j0 += CH) {
            T x[CH], rj[CH];
#pragma unroll
            for (int e = 0; e < CH; e++) {
                const int j = min(j0 + e, nj - 1);
                x[e] = c[2 * HT * j];
                rj[e] = r[HT * j + t];
            }
#pragma unroll
            for (int e = 0; e < CH; e++) {
                const int j = j0 + e;
                if (j < nj) {
                    q = (x[e] - (j == 0 ? T(0) : a1) * q) * rj[e];
                    c[2 * HT * j] = q;
                }
            }
        }
        c[2 * HT * (nj - 1)] = last;
        T s = last;
        for (int j0 = nj - 2; j0 >= 0; j0 -= CH) {
            T x[CH], f[CH];
#pragma unroll
            for (int e = 0; e < CH; e++) {
                const int j = max(j0 - e, 0);
                x[e] = c[2 * HT * j];
                f[e] = pf[HT * j + t];
            }
#pragma unroll
            for (int e = 0; e < CH; e++) {
                const int j = j0 - e;
                if (j >= 0) {
                    s = f[e] * s + x[e];
                    c[2 * HT * j] = s;
                }
            }
        }
    }
    __syncthreads();
    for (int w = threadIdx.x; w < HT * nj; w += HT_THREADS) {
        const int j = w / HT, t = w % HT;
        if (t >= nt) continue;
        T2 o;
        o.x = v[2 * w];
        o.y = v[2 * w + 1];
        h.spec2[(long)j * nx + i0 + t] = o;
    }
}

template <typename T>
__global__ void __launch_bounds__(HT_THREADS) k_hyd_thomas(KParams<T> p, HydArgs<T> h)
{
    extern __shared__ unsigned char hyd_smem[];
    // (lines too long for shared memory use a device buffer)
    if (h.tw) hyd_thomas_body(p, h, h.tw + (size_t)blockIdx.x * 4 * HT * p.ny);
    else hyd_thomas_body(p, h, (T *)hyd_smem);
}

// hydrostatic_pressure (pressure.cpp:453-537) from the current theta (and
// moisture), its density-weighted column average into level 0, the lid
// pressure (:285-286) into level NZ-1, and the total (:293-296)
template <typename T>
__global__ void __launch_bounds__(HC_THREADS) k_hyd_pi(KParams<T> p, KFields<T> F, HydArgs<T> h)
{
    extern __shared__ unsigned char hyd_smem[];
    const int nyi = p.ny - 2, nz = p.nz, lane = threadIdx.x & 31;
    T *g = (T *)hyd_smem;   // [HC][nz]: theta (times the water loading) / tbv^2, then the integral
    T *ps = g + HC * nz;    // [HC][nz]: the integral's steps
    T *wt = ps + HC * nz;   // [nz]: rhou tbv
    T *dzu = wt + nz;       // [nz]
    T *dzw = dzu + nz;      // [nz]
    const int ncol = (p.nx - 2) * nyi, col0 = blockIdx.x * HC;
    const T *TH = F.cur[FTH], *QV = F.cur[FQV], *QC = F.cur[FQC], *QR = F.cur[FQR];
    T *PI = F.pi;
    const T gcp = T(9.8 / 1004.0);
    for (int k = threadIdx.x; k < nz; k += HC_THREADS) {
        wt[k] = p.rhou[k] * p.tbv[k];
        dzu[k] = h.dzu[k];
        dzw[k] = h.dzw[k];
    }
    for (int cl = threadIdx.x >> 5; cl < HC && col0 + cl < ncol; cl += HC_WARPS) {
        const int col = col0 + cl, ci = col / nyi;
        const long c0 = gix(p.ny, nz, 1 + ci, 1 + col - ci * nyi, 0);
        T *gc = g + cl * nz, *pc = ps + cl * nz;
        for (int k = 1 + lane; k < nz - 1; k += 32) {
            const long c = c0 + k;
            T fac = p.moist ? (T(1.) + T(0.61) * QV[c] - QC[c] - QR[c]) : T(1);
            if (p.ice) fac = fac - F.cur[FQS][c] - F.cur[FQI][c];  // pressure.cpp:459-475
            gc[k] = (TH[c] * fac) / (p.tbv[k] * p.tbv[k]);
        }
        __syncwarp();
        // the steps of the downward integral, without the layer's depth
        for (int k = 1 + lane; k < nz - 1; k += 32)
            pc[k] = k == nz - 2 ? T(0.5) * gcp * gc[k] : T(0.5) * gcp * (gc[k + 1] + gc[k]);
    }
    __syncthreads();
    const int cl = threadIdx.x, col = col0 + cl;
    if (cl < HC && col < ncol) {
        const int ci = col / nyi, i = 1 + ci, j = 1 + col - ci * nyi;
        const T *__restrict__ st = ps + cl * nz;  // the steps; the integral replaces the loads in g
        T *__restrict__ pc = g + cl * nz;
        T up = -st[nz - 2] * dzw[nz - 1];
        pc[nz - 2] = up;
#pragma unroll 8
        for (int k = nz - 3; k > 0; k--) {
            up = fma_(-st[k], dzw[k + 1], up);
            pc[k] = up;
        }
        T avg = T(0), zsum = T(0);
#pragma unroll 8
        for (int k = 1; k < nz - 1; k++) {
            avg = fma_(mul_(wt[k], pc[k]), dzu[k], avg);
            zsum += dzu[k];
        }
        avg /= zsum;
        pc[0] = avg;
        pc[nz - 1] = (h.div[(long)i * p.ny + j] - avg) / h.rhoavg;
    }
    __syncthreads();
    for (int c2 = threadIdx.x >> 5; c2 < HC && col0 + c2 < ncol; c2 += HC_WARPS) {
        const int cc = col0 + c2, ci = cc / nyi;
        const T *pc = g + c2 * nz;
        const T lid = pc[nz - 1];
        // levels 1..NZ-2 to the edges that mirror the column as well
        with_mirrors(p.nx, p.ny, 1 + ci, 1 + cc - ci * nyi, [&](int i, int j) {
            const bool edge = i == 0 || j == 0 || i == p.nx - 1 || j == p.ny - 1;
            T *o = PI + gix(p.ny, nz, i, j, 0);
            for (int k = lane; k < nz; k += 32) {
                if (k == 0 || k == nz - 1) {
                    if (!edge) o[k] = pc[k];
                } else {
                    o[k] = pc[k] + lid;
                }
            }
        });
    }
}

// the pressure-gradient force of integrate_hydro (solver.cpp:70-79) over
// [1,N-1) x [1,N-1) x [1,NZ-1)
template <typename T>
__global__ void __launch_bounds__(256) k_hyd_project(KParams<T> p, KFields<T> F, T step)
{
    const int nzi = p.nz - 2, nyi = p.ny - 2;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;  // fewer than 2^31 points
    if (t >= (unsigned)((p.nx - 2) * nyi * nzi)) return;
    const int col = (int)t / nzi, k = 1 + (int)t - col * nzi, i = 1 + col / nyi, j = 1 + col % nyi;
    const long c = gix(p.ny, p.nz, i, j, k), sx = (long)p.ny * p.nz, sy = p.nz;
    const T *PI = F.pi;
    F.P[FU][c] = F.P[FU][c] - step * (p.dtx * T(1004) * p.tbv[k] * (PI[c] - PI[c - sx]));
    F.P[FV][c] = F.P[FV][c] - step * (p.dty * T(1004) * p.tbv[k] * (PI[c] - PI[c - sy]));
}

// w_velocity_LH (solver.cpp:144-163) into the current w
template <typename T>
__global__ void __launch_bounds__(HC_THREADS) k_hyd_w(KParams<T> p, KFields<T> F, HydArgs<T> h)
{
    extern __shared__ unsigned char hyd_smem[];
    const int nyi = p.ny - 2, nz = p.nz, lane = threadIdx.x & 31;
    T *dv = (T *)hyd_smem;   // [HC][nz]: the convergence term of level k (the level above its cell)
    T *ws = dv + HC * nz;    // [HC][nz]: w
    T *ra = ws + HC * nz;    // [nz]: rhow[k-1]/rhow[k]
    T *rb = ra + nz;         // [nz]: rhou[k-1]/rhow[k]
    const int ncol = (p.nx - 2) * nyi, col0 = blockIdx.x * HC;
    const T *UP = F.P[FU], *VP = F.P[FV];
    const long sx = (long)p.ny * nz, sy = nz;
    for (int k = 2 + threadIdx.x; k < nz - 1; k += HC_THREADS) {
        ra[k] = p.rhow[k - 1] / p.rhow[k];
        rb[k] = p.rhou[k - 1] / p.rhow[k];
    }
    __syncthreads();
    for (int cl = threadIdx.x >> 5; cl < HC && col0 + cl < ncol; cl += HC_WARPS) {
        const int col = col0 + cl, ci = col / nyi;
        const long c0 = gix(p.ny, nz, 1 + ci, 1 + col - ci * nyi, 0);
        for (int k = 2 + lane; k < nz - 1; k += 32) {
            const long c = c0 + k - 1;
            const T d = -(UP[c + sx] - UP[c]) * p.one_d_dx - (VP[c + sy] - VP[c]) * p.one_d_dy;
            dv[cl * nz + k] = rb[k] * d * h.dz / p.mu[k - 1];
        }
    }
    __syncthreads();
    const int cl = threadIdx.x;
    if (cl < HC && col0 + cl < ncol) {
        T *__restrict__ wc = ws + cl * nz;
        const T *__restrict__ dc = dv + cl * nz;
        wc[0] = T(0);
        wc[1] = T(0);
        wc[nz - 1] = T(0);
        T w = T(0);
#pragma unroll 8
        for (int k = 2; k < nz - 1; k++) {
            w = fma_(ra[k], w, dc[k]);
            wc[k] = w;
        }
    }
    __syncthreads();
    T *W = F.cur[FW];
    for (int c2 = threadIdx.x >> 5; c2 < HC && col0 + c2 < ncol; c2 += HC_WARPS) {
        const int cc = col0 + c2, ci = cc / nyi;
        T *o = W + gix(p.ny, nz, 1 + ci, 1 + cc - ci * nyi, 0);
        for (int k = lane; k < nz; k += 32) o[k] = ws[c2 * nz + k];
    }
}

}  // namespace ga
