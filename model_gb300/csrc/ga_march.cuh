// ---------------------------------------------------------------------------
// k_advect_march: the FP32 advection (advection.cpp:304-497 with the face
// fluxes of fluxes.cpp) for a horizontally uniform basic state and NZ % 4 == 0,
// marching along x.
//
// A block owns TJ interior columns of y, every level, a chunk of LI columns of
// x, and one field (a job); a thread owns one column and an aligned quad of
// four levels, and steps through the chunk.  For a fixed i the columns
// j0-3 .. j0+TJ+2 of a field are one contiguous run, so a plane arrives in
// shared memory as 16-byte asynchronous copies, two planes ahead of the step
// that needs it, in a ring of eight planes: the six-point stencils of both
// horizontal faces and the column neighbours of the top face read the ring.
// Each face is evaluated once: the west face is the previous step's east face
// (registers), the south face comes from the next thread row and the face
// below a quad from the next quad (shared memory, one exchange a step).  The
// first thread row evaluates only the north face south of the tile.
//
// Why one field per block: k_advect_quad passes two fields' faces of a 4x8
// tile through shared memory, evaluates 3.5 faces a cell in padded loops and
// reads 11 quads a face from L1.  Here the faces stay in registers, a plane is
// fetched once, both faces' arithmetic runs on packed pairs of levels
// (fma.rn.f32x2, half the instructions of scalar code), and fields run as
// separate blocks, which gives a small grid enough of them.  Bound: latency
// (all fields of a stage at 128x128x48, 49.6 us cold: issue 39% active, L1 51%,
// stalls an issue on loads 3.5, fixed latency 1.6, barriers 1.0).  Small grids
// run two blocks of 128 registers an SM (64x64x40 17 against 20 us a stage at
// three blocks of 80), large ones three, although at 80 registers a thread
// spills 304 bytes of stores and 184 of loads (512x512x64 820 against 870 us;
// 814 cold: issue 47%, L1 66%, stalls on loads 6.0).  All fields of a stage,
// against k_advect_quad's best tile: 64x64x40 21.5 -> 14.9 us, 128x128x48 67 ->
// 47 us, 512x512x64 1022 -> 820 us.
//
// Per level the arithmetic is that of the k_advect_tile face and tendency
// functions, expression for expression.
// ---------------------------------------------------------------------------
#pragma once
#include "ga_quad.cuh"

namespace ga {

constexpr int AM_THREADS = 256;  // thread rows of NZ/4 lanes, TJ + 1 rows
constexpr int AM_RING = 8;       // planes: six of the stencil, two on their way

// jobs of a launch: field kinds 0-7 (aq_field), buoyancy, or the three
// moisture fields one after another (the clipping record's bits of a point
// come from all three)
enum { AM_WB = 8, AM_QALL = 9 };

// per-level rows of nz the kernel reads besides the basic-state table
enum {
    MT_WB1,                  // WBAR one level up
    MT_NDTZ,                 // -(dt/dz) mu
    MT_RW, MT_RW1, MT_ODR,   // rhow, rhow one level up, 1/rhou
    MT_TBU, MT_TBD, MT_QBU, MT_QBD,  // steps of the base profiles above and below a level
    MT_QB0,                  // base humidity
    MT_RHOU, MT_VTD,         // density, fall-speed density factor
    MT_TBV,                  // virtual base temperature
    MT_TBVM,                 // and one level down
    MT_COUNT
};
static __global__ void k_march_table(KParams<float> p, float *t)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x, nz = p.nz;
    if (k >= nz) return;
    const int ku = min(k + 1, nz - 1), kd = max(k - 1, 0);
    t[MT_WB1 * nz + k] = p.btab[BT_WB * nz + ku];
    t[MT_NDTZ * nz + k] = -mul_(p.dtz, p.mu[k]);
    t[MT_RW * nz + k] = p.rhow[k];
    t[MT_RW1 * nz + k] = p.rhow[ku];
    t[MT_ODR * nz + k] = p.one_d_rhou[k];
    t[MT_TBU * nz + k] = p.tb[ku] - p.tb[k];
    t[MT_TBD * nz + k] = p.tb[k] - p.tb[kd];
    t[MT_QBU * nz + k] = p.qb[ku] - p.qb[k];
    t[MT_QBD * nz + k] = p.qb[k] - p.qb[kd];
    t[MT_QB0 * nz + k] = p.qb[k];
    t[MT_RHOU * nz + k] = p.rhou[k];
    t[MT_VTD * nz + k] = sqrt(p.rhou1 / p.rhou[k]);
    t[MT_TBV * nz + k] = p.tbv[k];
    t[MT_TBVM * nz + k] = p.tbv[kd];
}

// two FP32 values in a 64-bit register and their packed operations (each
// lane rounds as the scalar intrinsic)
typedef unsigned long long u64;
__device__ __forceinline__ u64 pk(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ u64 pk1(float a) { return pk(a, a); }
__device__ __forceinline__ void up(u64 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b)
{
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// +c where the lane of x is positive, -c elsewhere (also at 0): the sign bit
// of 0 - x is set exactly where x > 0.  nc is the bit pattern of -c in both lanes
__device__ __forceinline__ u64 upwind2(u64 x, u64 nc)
{
    return (sub2(0ull, x) & 0x8000000080000000ull) ^ nc;
}
// levels k0, k0+1 in a, k0+2, k0+3 in b
struct P4 {
    u64 a, b;
};
__device__ __forceinline__ P4 ldsp(const float *a)
{
    const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(a);
    return P4{t.x, t.y};
}
__device__ __forceinline__ P4 ldgp(const float *a)
{
    const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2 *>(a));
    return P4{t.x, t.y};
}
__device__ __forceinline__ void stsp(float *a, const P4 &v)
{
    *reinterpret_cast<ulonglong2 *>(a) = make_ulonglong2(v.a, v.b);
}
// the faces of two levels: face5_cs, face3_cs
__device__ __forceinline__ u64 face5_2(u64 am2, u64 am1, u64 a0, u64 a1, u64 a2, u64 a3, u64 cs)
{
    const u64 c6 = fma2(pk1(W<float>::c1_60), add2(a3, am2),
                        fma2(pk1(-W<float>::c2_15), add2(a2, am1), mul2(pk1(W<float>::c37_60), add2(a1, a0))));
    const u64 u5 = fma2(pk1(-10.f), sub2(a1, a0), fma2(pk1(5.f), sub2(a2, am1), sub2(am2, a3)));
    return fma2(cs, u5, c6);
}
__device__ __forceinline__ u64 face3_2(u64 am1, u64 a0, u64 a1, u64 a2, u64 cs)
{
    const u64 c4 = fma2(pk1(-W<float>::c1_12), add2(a2, am1), mul2(pk1(W<float>::c7_12), add2(a1, a0)));
    const u64 u3 = fma2(pk1(-3.f), sub2(a1, a0), sub2(a2, am1));
    return fma2(cs, u3, c4);
}
__device__ __forceinline__ u64 flux2_2(u64 a, u64 b, u64 c, u64 d) { return fma2(a, b, mul2(c, d)); }

// tile of a launch: TJ columns of y and LI of x per block, and the tile counts
struct MarchGeom {
    int tj, li, njt, nit;
};
// TJ: as many thread rows as fit AM_THREADS, the tiles of a row of equal size.
// LI: a chunk starts with six planes to fetch and one extra east face, so it
// is as long as leaves about six blocks for each SM (three waves of two blocks
// or two of three), at least 4 and at most 16 columns: 64x64x40 took 15 us a stage with 4 and 24 with 8,
// 128x128x48 49 with 5 and 64 with 16 (all fields, one stream); at 512x512x64
// 16 and 32 are equal.  li > 0 fixes it.
__host__ inline MarchGeom march_geom(int nx, int ny, int nz, int njobs, int nsm, int li = 0)
{
    MarchGeom g;
    const int tjm = std::max(1, AM_THREADS / (nz / 4) - 1);
    g.njt = (ny - 6 + tjm - 1) / tjm;
    g.tj = (ny - 6 + g.njt - 1) / g.njt;
    const long cols = (long)(nx - 6) * g.njt * njobs;
    g.li = li > 0 ? li : (int)std::min(16L, std::max(4L, cols / (6L * nsm)));
    g.nit = (nx - 6 + g.li - 1) / g.li;
    g.li = (nx - 6 + g.nit - 1) / g.nit;
    return g;
}
// The blocks of one job next to each other while ten fields of the grid fit
// L2 (an SM then runs one instruction stream at a time and the winds are read
// from L2 by every job: 128x128x48 49 against 52 us a stage); the jobs of one
// tile next to each other on larger grids, where each job would read the winds
// from DRAM again (512x512x64 820 against 955 us).
__host__ inline bool march_by_job(long n) { return (size_t)n * sizeof(float) * 10 <= ((size_t)96 << 20); }
__host__ inline size_t march_smem(int tj, int nz)
{
    return ((size_t)AM_RING * (tj + 6) * nz + 8 + (size_t)(tj + 1) * nz + (size_t)(tj + 1) * (nz / 4)) * sizeof(float);
}

__device__ __forceinline__ void cp16(float *dst, const float *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// classes of fields that share one instruction stream
enum { MC_U, MC_V, MC_BASE, MC_PLAIN, MC_FALL };

// field kind fk over the block's tile; every thread of the block calls it.
// BASE: theta and qv, with a basic-state part; PLAIN: cloud water; FALL: rain,
// snow, ice.
template <int C>
__device__ __forceinline__ void march_field(const KParams<float> &p, const KFields<float> &F, float *sm, int tjg,
                                            int fk, int i0, int li, int j0, int tj, float step, int what)
{
    const int nz = p.nz, NQ = nz >> 2, sx = p.ny * nz, sy = nz;
    const int tid = threadIdx.x, jj = tid / NQ, q = tid - jj * NQ, k0 = 4 * q;
    const bool row = jj <= tj, cell = row && jj >= 1;  // jj = 0: the row south of the tile
    const bool qlo = q == 0, qhi = q == NQ - 1;
    const int j = j0 - 1 + jj;
    const int plane = (tj + 6) * nz, nchunk = plane >> 2;
    float *nf = sm + AM_RING * (tjg + 6) * nz + 8, *tf = nf + (tjg + 1) * nz;
    const int XF = C == MC_U ? FU : C == MC_V ? FV : aq_field(fk);
    const float *X = F.cur[XF], *U = F.cur[FU], *V = F.cur[FV], *Wc = F.cur[FW], *Mf = F.M[XF];
    float *Pf = F.P[XF];
    const float *btab = p.btab, *mtab = p.mtab;
    const int br = fk == 3 ? 1 : 0;  // BASE: the basic-state rows of qv
    // table rows at this thread's quad
    const int o_ub = (C <= MC_V ? BT_UA : BT_UB) * nz, o_vb = (C <= MC_V ? BT_VA : BT_VB) * nz;
    const int o_c6 = (C == MC_U ? BT_C6_UB : C == MC_V ? BT_C6_VB : BT_C6_THB + br) * nz;
    const int o_c4 = (C == MC_U ? BT_C4_UB : C == MC_V ? BT_C4_VB : BT_C4_THB + 2 * br) * nz;
    const int o_h2 = (C == MC_U ? BT_H2_UB : C == MC_V ? BT_H2_VB : BT_H2_THB + br) * nz;
    auto bt = [&](int o) { return ldgp(btab + (o + k0)); };
    auto mt = [&](int r) { return ldgp(mtab + (r * nz + k0)); };
    const u64 n60 = pk1(-W<float>::c1_60), n12 = pk1(-W<float>::c1_12), half = pk1(0.5f);
    const int xg = (j0 - 3) * nz + 4 * tid;
    auto fetch = [&](int i) {
        float *dst = sm + (i & (AM_RING - 1)) * plane + 4 * tid;
        const float *src = X + (i * sx + xg);
        if (tid < nchunk) cp16(dst, src);
        if (tid + AM_THREADS < nchunk) cp16(dst + 4 * AM_THREADS, src + 4 * AM_THREADS);
    };
    const int ilast = i0 + li + 2;  // the last plane a step reads
    __syncthreads();                // the ring and exchanges of an earlier field are free
#pragma unroll 1
    for (int i = i0 - 3; i <= i0 + 2; i++) fetch(i);
    cp_commit();
    if (i0 + 3 <= ilast) fetch(i0 + 3);
    cp_commit();

    const int xo = (jj + 2) * nz + k0;  // this column's quad in a plane
    auto slot = [&](int i) { return (i & (AM_RING - 1)) * plane + xo; };
    int w0 = slot(i0 - 3), w1 = slot(i0 - 2), w2 = slot(i0 - 1), w3 = slot(i0), w4 = slot(i0 + 1),
        w5 = slot(i0 + 2);  // planes i-2 .. i+3
    P4 ew{0, 0};              // west face
    P4 a0{0, 0}, a1{0, 0};    // the other wind at the last step (u: v at i-1; v: u at i), columns j and j+-1
    const float dtf = row && C <= MC_V ? mul_(p.dt, p.f[j]) : 0.f;
    const u64 cor = pk1(C == MC_U ? dtf : -dtf);
    int c = gix(p.ny, nz, i0 - 1, j, k0);
#pragma unroll 1
    for (int i = i0 - 1; i < i0 + li; i++, c += sx) {
        cp_wait<1>();      // plane i+3 of this thread
        __syncthreads();   // of every thread; and plane i-3 and the exchanges are no longer read
        if (i + 5 <= ilast) fetch(i + 5);
        cp_commit();
        const bool first = i < i0;
        P4 ee{0, 0}, nn{0, 0}, tt{0, 0}, m{0, 0}, b0{0, 0}, b1{0, 0};
        float wv[5];  // w at levels k0 .. k0+4
        if (cell) {
            // the step's global loads before its arithmetic
            P4 ua{0, 0}, ub{0, 0};
            if (C != MC_U) ua = ldgp(U + c + sx);
            if (C == MC_V) ub = ldgp(U + c + sx - sy);
            if (C == MC_U) {  // v of column i: the Coriolis term and the north face
                b0 = ldgp(V + c);
                b1 = ldgp(V + c + sy);
            }
            if (!first) {
                m = ldgp(Mf + c);
                const P4 wq = ldgp(Wc + c);
                up(wq.a, wv[0], wv[1]);
                up(wq.b, wv[2], wv[3]);
                wv[4] = qhi ? 0.f : __ldg(Wc + c + 4);
            }
            // ---- east face between i and i+1
            const P4 x0 = ldsp(sm + w0), x1 = ldsp(sm + w1), x2 = ldsp(sm + w2), x3 = ldsp(sm + w3), x4 = ldsp(sm + w4),
                     x5 = ldsp(sm + w5);
            const P4 ubar = bt(o_ub);
            P4 c6{0, 0};
            if (C <= MC_BASE) c6 = bt(o_c6);
            auto east = [&](u64 X0, u64 X1, u64 X2, u64 X3, u64 X4, u64 X5, u64 A, u64 B, u64 ubr, u64 c6r) {
                if (C <= MC_V) {
                    const u64 av = mul2(half, C == MC_U ? add2(X3, X2) : add2(A, B)), at = add2(ubr, av);
                    return flux2_2(av, c6r, at, face5_2(X0, X1, X2, X3, X4, X5, upwind2(at, n60)));
                }
                const u64 at = add2(ubr, A), f = face5_2(X0, X1, X2, X3, X4, X5, upwind2(at, n60));
                return C == MC_BASE ? flux2_2(A, c6r, at, f) : mul2(at, f);
            };
            ee.a = east(x0.a, x1.a, x2.a, x3.a, x4.a, x5.a, ua.a, ub.a, ubar.a, c6.a);
            ee.b = east(x0.b, x1.b, x2.b, x3.b, x4.b, x5.b, ua.b, ub.b, ubar.b, c6.b);
            if (C == MC_V) { b0 = ua; b1 = ub; }
        }
        if (row && !first) {
            // ---- north face between j and j+1
            P4 va{0, 0}, vb{0, 0};
            if (C == MC_U) {
                va = cell ? b1 : ldgp(V + c + sy);
                vb = cell ? a1 : ldgp(V + c - sx + sy);
            } else if (C != MC_V) {
                va = ldgp(V + c + sy);
            }
            const float *xp = sm + w2;
            const P4 x0 = ldsp(xp - 2 * nz), x1 = ldsp(xp - nz), x2 = ldsp(xp), x3 = ldsp(xp + nz),
                     x4 = ldsp(xp + 2 * nz), x5 = ldsp(xp + 3 * nz);
            const P4 vbar = bt(o_vb);
            P4 c6{0, 0};
            if (C <= MC_BASE) c6 = bt(o_c6);
            auto north = [&](u64 X0, u64 X1, u64 X2, u64 X3, u64 X4, u64 X5, u64 A, u64 B, u64 vbr, u64 c6r) {
                if (C <= MC_V) {
                    const u64 av = mul2(half, C == MC_U ? add2(A, B) : add2(X3, X2)), at = add2(vbr, av);
                    return flux2_2(av, c6r, at, face5_2(X0, X1, X2, X3, X4, X5, upwind2(at, n60)));
                }
                const u64 at = add2(vbr, A), f = face5_2(X0, X1, X2, X3, X4, X5, upwind2(at, n60));
                return C == MC_BASE ? flux2_2(A, c6r, at, f) : mul2(at, f);
            };
            nn.a = north(x0.a, x1.a, x2.a, x3.a, x4.a, x5.a, va.a, vb.a, vbar.a, c6.a);
            nn.b = north(x0.b, x1.b, x2.b, x3.b, x4.b, x5.b, va.b, vb.b, vbar.b, c6.b);
            stsp(nf + jj * nz + k0, nn);
            if (cell) {
                // ---- top faces between k and k+1, k = k0 .. k0+3; 2nd order at
                // k = 1 and NZ-2, none at 0 and NZ-1.  Values beyond the column
                // are neighbouring ones that no kept result uses.
                float xv[7];  // levels k0-1 .. k0+5
                xv[0] = xp[-1];
                up(x2.a, xv[1], xv[2]);
                up(x2.b, xv[3], xv[4]);
                xv[5] = xp[4];
                xv[6] = xp[5];
                const u64 o0 = pk(xv[0], xv[1]), o1 = pk(xv[2], xv[3]), o2 = pk(xv[4], xv[5]), e2 = pk(xv[5], xv[6]);
                const u64 wa_ = pk(wv[1], wv[2]), wb_ = pk(wv[3], wv[4]);  // w one level up
                float f4[4];
                if (C <= MC_BASE) {
                    const P4 wbar = C <= MC_V ? bt(BT_WA * nz) : mt(MT_WB1), h2 = bt(o_h2), c4 = bt(o_c4), u3 = bt(o_c4 + nz);
                    u64 av[2] = {wa_, wb_};
                    if (C <= MC_V) {  // averaged with the second w, column i-1 (u) or j-1 (v)
                        const int o2w = C == MC_U ? -sx : -sy;
                        const P4 wq = ldgp(Wc + c + o2w);
                        float y0, y1, y2, y3;
                        up(wq.a, y0, y1);
                        up(wq.b, y2, y3);
                        const float y4 = qhi ? 0.f : __ldg(Wc + c + o2w + 4);
                        av[0] = mul2(half, add2(wa_, pk(y1, y2)));
                        av[1] = mul2(half, add2(wb_, pk(y3, y4)));
                    }
                    const u64 at0 = add2(wbar.a, av[0]), at1 = add2(wbar.b, av[1]);
                    u64 xt0 = face3_2(o0, x2.a, o1, x2.b, upwind2(at0, n12));
                    u64 xt1 = face3_2(o1, x2.b, o2, e2, upwind2(at1, n12));
                    u64 xb0 = fma2(upwind2(av[0], n12), u3.a, c4.a), xb1 = fma2(upwind2(av[1], n12), u3.b, c4.b);
                    if (qlo) {  // k = 1
                        xt0 = mul2(half, add2(o1, x2.a));
                        xb0 = h2.a;
                    }
                    if (qhi) {  // k = NZ-2
                        xt1 = mul2(half, add2(o2, x2.b));
                        xb1 = h2.b;
                    }
                    tt.a = flux2_2(av[0], xb0, at0, xt0);
                    tt.b = flux2_2(av[1], xb1, at1, xt1);
                } else {
                    const P4 wbar = mt(MT_WB1);
                    u64 at0 = add2(wbar.a, wa_), at1 = add2(wbar.b, wb_);
                    float vt[5];
                    if (C == MC_FALL) {
                        // fall speeds at levels k0 .. k0+4, from the rain itself
                        // (Eulerian Kessler fallout, whose values the step
                        // keeps) or stored by their own kernel
                        float *fa = fk == 5 ? F.vt : fk == 6 ? F.sts : F.its;
                        const bool own = fk == 5 && p.rf == 1 && !p.ice;
                        const float *r_rho = mtab + (MT_RHOU * nz + k0), *r_vtd = mtab + (MT_VTD * nz + k0);
#pragma unroll
                        for (int e = 0; e < 5; e++) {
                            float v = 0.f;
                            if (own && !(qhi && e >= 3)) {
                                // level 0 takes level 1's value
                                const float qr = e == 0 && qlo ? xv[2] : xv[e + 1];
                                const int ke = e == 0 && qlo ? 1 : e;
                                if (qr > 1.0e-12f) {  // fall_speed_point
                                    const float qrr = fmax(qr * 0.001f * __ldg(r_rho + ke), 0.0f);
                                    v = 36.34f * (pow(qrr, 0.1364f)) * __ldg(r_vtd + ke);
                                }
                            } else if (!(qhi && e == 4)) {
                                v = fa[c + e];
                            }
                            vt[e] = v;
                        }
                        if (own) {  // the advected cells' speeds
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if (!(qhi && e == 3)) fa[c + e] = vt[e];
                        }
                        at0 = sub2(at0, mul2(half, add2(pk(vt[0], vt[1]), pk(vt[1], vt[2]))));
                        at1 = sub2(at1, mul2(half, add2(pk(vt[2], vt[3]), pk(vt[3], vt[4]))));
                    }
                    u64 xt0 = face3_2(o0, x2.a, o1, x2.b, upwind2(at0, n12));
                    u64 xt1 = face3_2(o1, x2.b, o2, e2, upwind2(at1, n12));
                    if (qlo) xt0 = mul2(half, add2(o1, x2.a));
                    if (qhi) xt1 = mul2(half, add2(o2, x2.b));
                    tt.a = mul2(at0, xt0);
                    tt.b = mul2(at1, xt1);
                    if (C == MC_FALL && qlo) {  // the outflow through the ground
                        const float s0 = 0.5f * (xv[1] + xv[2]);
                        float u0, u1;
                        up(tt.a, u0, u1);
                        tt.a = pk(-0.5f * (vt[1] + vt[0]) * s0, u1);
                    }
                }
                up(tt.a, f4[0], f4[1]);
                up(tt.b, f4[2], f4[3]);
                if (C != MC_FALL && qlo) tt.a = pk(0.f, f4[1]);
                if (qhi) {
                    f4[3] = 0.f;
                    tt.b = pk(f4[2], 0.f);
                }
                tf[jj * NQ + q] = f4[3];
            }
        }
        if (!first) __syncthreads();
        if (cell && !first) {
            const P4 ns = ldsp(nf + (jj - 1) * nz + k0);
            const float tb0 = qlo ? 0.f : tf[jj * NQ + q - 1];
            const P4 ndtz = mt(MT_NDTZ), rw = mt(MT_RW), rw1 = mt(MT_RW1),
                     odr = mt(MT_ODR);
            float t0, t1, t2, t3;
            up(tt.a, t0, t1);
            up(tt.b, t2, t3);
            const u64 ndx = pk1(-p.dtx), ndy = pk1(-p.dty), st = pk1(step);
            // flux_div
            auto div = [&](u64 E, u64 Ew, u64 Nn, u64 Ns, u64 T, u64 Tl, u64 nd, u64 r0, u64 r1, u64 od) {
                const u64 w = fma2(r0 ^ 0x8000000080000000ull, Tl, mul2(r1, T));
                return fma2(mul2(nd, w), od, fma2(ndy, sub2(Nn, Ns), mul2(ndx, sub2(E, Ew))));
            };
            u64 d0 = div(ee.a, ew.a, nn.a, ns.a, tt.a, pk(tb0, t0), ndtz.a, rw.a, rw1.a, odr.a);
            u64 d1 = div(ee.b, ew.b, nn.b, ns.b, tt.b, pk(t1, t2), ndtz.b, rw.b, rw1.b, odr.b);
            if (C <= MC_V) {
                // 0.25 * the four surrounding winds, in the reference's order
                const u64 qt = pk1(0.25f);
                const u64 s0 = C == MC_U ? add2(add2(add2(b0.a, b1.a), a0.a), a1.a)
                                         : add2(add2(add2(a0.a, b0.a), a1.a), b1.a);
                const u64 s1 = C == MC_U ? add2(add2(add2(b0.b, b1.b), a0.b), a1.b)
                                         : add2(add2(add2(a0.b, b0.b), a1.b), b1.b);
                d0 = fma2(cor, mul2(qt, s0), d0);
                d1 = fma2(cor, mul2(qt, s1), d1);
            } else if (C == MC_BASE) {  // sub_base
                const P4 bu = mt(br ? MT_QBU : MT_TBU), bd = mt(br ? MT_QBD : MT_TBD);
                const u64 z0 = fma2(mul2(rw1.a, pk(wv[1], wv[2])), bu.a, mul2(mul2(rw.a, pk(wv[0], wv[1])), bd.a));
                const u64 z1 = fma2(mul2(rw1.b, pk(wv[3], wv[4])), bu.b, mul2(mul2(rw.b, pk(wv[2], wv[3])), bd.b));
                d0 = fma2(ndtz.a, mul2(mul2(half, z0), odr.a), d0);
                d1 = fma2(ndtz.b, mul2(mul2(half, z1), odr.b), d1);
            }
            Q4 r;
            const u64 v0 = fma2(st, d0, m.a), v1 = fma2(st, d1, m.b);
            up(v0, r.v[0], r.v[1]);
            up(v1, r.v[2], r.v[3]);
            if (C >= MC_BASE && (what & ADV_ZERO) && fk >= 3) {  // zero_moisture (microphysics.cpp:675-700)
                unsigned bits = 0;
                if (C == MC_BASE) {
                    const Q4 qbar = ldg4(btab, BT_QB * nz + k0), qb0 = ldg4(mtab, MT_QB0 * nz + k0);
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (r.v[e] + qbar.v[e] + qb0.v[e] < 0) {
                            r.v[e] = -(qbar.v[e] + qb0.v[e]);
                            bits |= 1u << e;
                        }
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (r.v[e] < 0) {
                            r.v[e] = 0;
                            bits |= 1u << e;
                        }
                }
                if (F.qmask && fk <= 5) {
                    unsigned char *qm = F.qmask + c;
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const unsigned char b = (unsigned char)((bits >> e) & 1u);
                        if ((qlo && e == 0) || (qhi && e == 3)) continue;
                        if (fk == 3) qm[e] = b;
                        else qm[e] |= (unsigned char)(b << (fk - 3));
                    }
                }
            }
            if (qlo) {  // levels 1 .. NZ-2
                Pf[c + 1] = r.v[1];
                Pf[c + 2] = r.v[2];
                if (!qhi) Pf[c + 3] = r.v[3];
            } else if (qhi) {
                Pf[c] = r.v[0];
                Pf[c + 1] = r.v[1];
                Pf[c + 2] = r.v[2];
            } else {
                stg4(Pf + c, r);
            }
        }
        ew = ee;
        a0 = b0;
        a1 = b1;
        w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5;
        w5 = slot(i + 4);
    }
}

// buoyancy overwrite of w (advection.cpp:329-337) over the block's tile
__device__ __forceinline__ void march_buoyancy(const KParams<float> &p, const KFields<float> &F, int i0, int li,
                                               int j0, int tj, float sdtg)
{
    const int nz = p.nz, NQ = nz >> 2;
    const int jj = threadIdx.x / NQ, q = threadIdx.x - jj * NQ, k0 = 4 * q;
    if (jj >= tj) return;
    const Q4 tq = ldg4(p.mtab, MT_TBV * nz + k0);
    const float tv[5] = {__ldg(p.mtab + MT_TBVM * nz + k0), tq.v[0], tq.v[1], tq.v[2], tq.v[3]};
    // levels k0-1 .. k0+3 of a field's column
    auto col = [&](const float *a, int c, float *o) {
        const Q4 v = ldg4(a, c);
        o[0] = k0 > 0 ? __ldg(a + c - 1) : 0.f;
#pragma unroll
        for (int e = 0; e < 4; e++) o[1 + e] = v.v[e];
    };
    for (int i = i0; i < i0 + li; i++) {
        const int c = gix(p.ny, nz, i, j0 + jj, k0);
        float th[5], bb[5];
        col(F.cur[FTH], c, th);
        const Q4 m = ldg4(F.M[FW], c);
        if (!p.moist) {
#pragma unroll
            for (int e = 0; e < 5; e++) bb[e] = th[e] / tv[e];
        } else {
            float qv[5], qc[5], qr[5];
            col(F.cur[FQV], c, qv);
            col(F.cur[FQC], c, qc);
            col(F.cur[FQR], c, qr);
#pragma unroll
            for (int e = 0; e < 5; e++) bb[e] = buoy_moist(th[e], tv[e], qv[e], qc[e], qr[e]);
        }
        if (p.ice) {  // buoyancy_cold_micro (advection.cpp:56-58): less ice, then snow
            float qi[5], qs[5];
            col(F.cur[FQI], c, qi);
            col(F.cur[FQS], c, qs);
#pragma unroll
            for (int e = 0; e < 5; e++) {
                bb[e] = bb[e] - qi[e];
                bb[e] = bb[e] - qs[e];
            }
        }
        Q4 r;
#pragma unroll
        for (int e = 0; e < 4; e++) r.v[e] = fma_(sdtg, add_(bb[e + 1], bb[e]), m.v[e]);
        aq_store(F.P[FW], c, k0, nz, 2, r);
    }
}

// tile (it, jt) of job `job` on geometry g; the batched ensemble kernel calls
// it per member
__device__ __forceinline__ void march_body(const KParams<float> &p, const KFields<float> &F, const MarchGeom &g,
                                           int job, int it, int jt, float step, float sdtg, int what)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *sm = (float *)smem_raw;
    const int i0 = 3 + it * g.li, j0 = 3 + jt * g.tj;
    const int li = min(g.li, p.nx - 3 - i0), tj = min(g.tj, p.ny - 3 - j0);
    if (job == AM_WB) {
        march_buoyancy(p, F, i0, li, j0, tj, sdtg);
        return;
    }
    const int f0 = job == AM_QALL ? 3 : job, f1 = job == AM_QALL ? 5 : job;
    for (int fk = f0; fk <= f1; fk++) {
        if (fk == 0) march_field<MC_U>(p, F, sm, g.tj, fk, i0, li, j0, tj, step, what);
        else if (fk == 1) march_field<MC_V>(p, F, sm, g.tj, fk, i0, li, j0, tj, step, what);
        else if (fk <= 3) march_field<MC_BASE>(p, F, sm, g.tj, fk, i0, li, j0, tj, step, what);
        else if (fk == 4) march_field<MC_PLAIN>(p, F, sm, g.tj, fk, i0, li, j0, tj, step, what);
        else march_field<MC_FALL>(p, F, sm, g.tj, fk, i0, li, j0, tj, step, what);
    }
}

// jobs: four bits each, job 0 lowest.  Grid (tiles of y, chunks of x, jobs)
// where `by_job` (the blocks of one field next to each other: one instruction
// stream at a time per SM), else (jobs, chunks, tiles)
template <int MB>
__global__ void __launch_bounds__(AM_THREADS, MB)
    k_advect_march(KParams<float> p, KFields<float> F, MarchGeom g, unsigned long long jobs, int by_job, float step,
                   float sdtg, int what)
{
    if (what & ADV_MIRROR) {  // mirror copies (edge points from non-advected ones), grid-stride
        const long nt = (long)gridDim.x * gridDim.y * gridDim.z * AM_THREADS;
        const long ntot = 2L * (p.nx + p.ny - 2) * (p.nz - 2);
        const long b = ((long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        for (long t = b * AM_THREADS + threadIdx.x; t < ntot; t += nt)
            mirror_edges_body(p, F.P[FU], F.P[FV], p.hydrostatic ? F.P[FV] : F.P[FW], t);
    }
    const int jb = by_job ? blockIdx.z : blockIdx.x, jt = by_job ? blockIdx.x : blockIdx.z;
    march_body(p, F, g, (int)((jobs >> (4 * jb)) & 15ull), blockIdx.y, jt, step, sdtg, what);
}

// the jobs of a launch mask
__host__ inline unsigned long long march_jobs(int what, bool record, int *njobs)
{
    unsigned long long j = 0;
    int n = 0;
    auto add = [&](int k) { j |= (unsigned long long)k << (4 * n++); };
    if (what & ADV_UV) { add(0); add(1); }
    if (what & ADV_TH) add(2);
    if (what & ADV_Q) {
        if (record) {
            add(AM_QALL);
        } else {
            add(5);  // the rain's fall speeds make it the longest
            add(3);
            add(4);
        }
    }
    if (what & ADV_ICE) { add(6); add(7); }
    if (what & ADV_WB) add(AM_WB);
    *njobs = n;
    return j;
}

}  // namespace ga
