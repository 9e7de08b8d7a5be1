// The sweeps, residual and CG update of a stretched 3D level in FP64 on the colour-split layout (nb_split.cu has the
// layout, the march and the transfers): the plain FP64 form's kernels on stretched grids.
//
// Stencil. Between cells of widths w and centre distances g the coefficient of a face is the product of the two other
// widths over the distance: w_x w_z / g_y along i, w_y w_z / g_x along j, w_x w_y / g_z along k. A thread's row j and
// its elements' k range stay fixed along the march, so the sum over the six neighbours is formed as
//   w_z (w_x (n_i+ / g + n_i- / g) + w_y (n_j+ / g + n_j- / g)) + w_x w_y (n_k+ / g + n_k- / g)
// with the x and z entries in registers and three y entries read per plane: ten FP64 operations a cell, where forming
// the six coefficients and the diagonal, and dividing by it, took about sixty. The diagonal and its reciprocal are
// kept per cell (dg, idg: built once per layout, zero off the unknowns); a sweep reads the reciprocal, the residual
// and the update the diagonal.
//
// With N = 2 elements a thread, k = 2m + q (q alternating with the plane): the face between k = 2m and 2m + 1 is
// every element's one toward the same m of the other colour (zc), the face on its other side is zs[q].
//
// The cylinder grid 192 x 128 x 128 to 1e-8 in FP64 (16 CG iterations, B200): 11.1 ms with one thread per cell and
// the coefficients formed per cell, 6.6 ms with these kernels.
#include "nb_quad.cuh"

namespace nb
{

namespace
{

constexpr int kN = kQ<double>;
using Q2 = Quad<double>;

// A thread's table entries along its row (x) and elements (z)
struct StRow
{
    double wx, gx0, gx1; // Width x of row j, 1/FaceGap x below and above it
    double wz[2][kN];    // Width z of k = 2m + q
    double zc[kN];       // 1/FaceGap z between k = 2m and 2m + 1
    double zs[2][kN];    // 1/FaceGap z on the other side of k = 2m + q
};

__device__ __forceinline__ StRow StRowOf(const LevelView &v, const QuadPos &P)
{
    StRow s;
    s.wx = v.w[0][P.j + 1];
    s.gx0 = v.igd[0][P.j];
    s.gx1 = v.igd[0][P.j + 1];
#pragma unroll
    for (int x = 0; x < kN; x++)
    {
        const int k = 2 * (P.m0 + x), last = v.Nz - 1; // past the row's end: padding, whose results are masked
        s.wz[0][x] = v.w[2][min(k, last) + 1];
        s.wz[1][x] = v.w[2][min(k + 1, last) + 1];
        s.zs[0][x] = v.igd[2][min(k, last + 1)];
        s.zc[x] = v.igd[2][min(k + 1, last + 1)];
        s.zs[1][x] = v.igd[2][min(k + 2, last + 1)];
    }
    return s;
}

// plane i's y entries
struct StPlane
{
    double wy, gLo, gHi, wxy;
};
__device__ __forceinline__ StPlane StPlaneOf(const LevelView &v, const StRow &s, int i)
{
    StPlane p;
    p.wy = v.w[1][i + 1];
    p.gLo = v.igd[1][i];
    p.gHi = v.igd[1][i + 1];
    p.wxy = s.wx * p.wy;
    return p;
}

// sum of coefficient times neighbour for element x: nP, nM along i, jp, jm along j, nC the other colour's element m,
// nS its shifted one
__device__ __forceinline__ double StSum(const StRow &s, const StPlane &p, int q, int x, double nP, double nM,
                                        double jp, double jm, double nC, double nS)
{
    const double wz = q ? s.wz[1][x] : s.wz[0][x], zs = q ? s.zs[1][x] : s.zs[0][x];
    return wz * (s.wx * (p.gHi * nP + p.gLo * nM) + p.wy * (s.gx1 * jp + s.gx0 * jm)) +
           p.wxy * (s.zc[x] * nC + zs * nS);
}

} // namespace

// ---- per layout: the diagonal and its reciprocal ----
__global__ void __launch_bounds__(256) k_stretched_diag(LevelView v, double *__restrict__ dg, double *__restrict__ idg)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < v.cells;
         c += (long long)gridDim.x * blockDim.x)
    {
        const unsigned code = v.code[c];
        if (!(code & CODE_UNKNOWN)) continue; // both arrays were zeroed
        const int k = (int)(c % v.Nz);
        const long long rr = c / v.Nz;
        const int j = (int)(rr % v.Nx), i = (int)(rr / v.Nx);
        const double ax = Wd(v, 1, i) * Wd(v, 2, k), ay = Wd(v, 0, j) * Wd(v, 2, k), az = Wd(v, 0, j) * Wd(v, 1, i);
        const double cq[6] = {ay / Gp(v, 1, i),     ay / Gp(v, 1, i - 1), ax / Gp(v, 0, j),
                              ax / Gp(v, 0, j - 1), az / Gp(v, 2, k),     az / Gp(v, 2, k - 1)};
        double d = 0.0;
        for (int q = 0; q < 6; q++)
            if (code >> q & 1u) d += cq[q];
        if (code & CODE_DIRICHLET)
            for (int q = 0; q < 6; q++)
            {
                if (!IsDirichlet(v.types[c + NbrOffset(v, q)])) continue;
                const int ni = i + (q == 0) - (q == 1), nj = j + (q == 2) - (q == 3), nk = k + (q == 4) - (q == 5);
                const int a = q < 2 ? 1 : (q < 4 ? 0 : 2), n = q < 2 ? i : (q < 4 ? j : k);
                // a ring neighbour's value sits on the face: FaceGap / (Width / 2), PressureSettings.h:307-310
                d += OnRing(v, ni, nj, nk) ? cq[q] * (Gp(v, a, (q & 1) ? n - 1 : n) / (0.5 * Wd(v, a, n))) : cq[q];
            }
        const long long o = VecIdx(v, i, j, k);
        dg[o] = d;
        idg[o] = d != 0.0 ? 1.0 / d : 0.0;
    }
}

void LaunchStretchedDiag(const LevelView &v, double *dg, double *idg, cudaStream_t st)
{
    const long long blocks = (v.cells + 255) / 256;
    NB_COUNT_LAUNCH();
    k_stretched_diag<<<(unsigned)(blocks < 148 * 8 ? (blocks > 0 ? blocks : 1) : 148 * 8), 256, 0, st>>>(v, dg, idg);
}

// ---- smoothing ----
// The first red-black sweep from a zero iterate: red e = r / diag, black e = (r + sum of the red neighbours) / diag
// with the red neighbours formed from r and the reciprocals.
__global__ void __launch_bounds__(kPairThreads, 3) k_stretched_first(LevelView v, const double *__restrict__ r,
                                                                    double *__restrict__ e)
{
    PdlWait();
    PdlTrigger();
    const Blk blk = ThisBlk();
    const QuadPos P = QuadStart<kN>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1)) return;
    const StRow S = StRowOf(v, P);
    const long long hb = v.sHalf;
    const double *R0 = r + P.off, *R1 = R0 + hb, *G0 = v.idg + P.off, *G1 = G0 + hb;
    double *X0 = e + P.off, *X1 = X0 + hb;
    auto red = [&](long long o) {
        Q2 a = LQ(R0 + o);
        const Q2 g = LQ(G0 + o);
#pragma unroll
        for (int x = 0; x < kN; x++) a.v[x] *= g.v[x];
        return a;
    };
    Q2 RM = red(-P.PS), RC = red(0);
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Q2 RP = red(o + P.PS), RJp = red(o + P.RS), RJm = red(o - P.RS);
        const Q2 rb = LQOnce(R1 + o), gb = LQ(G1 + o);
        const StPlane Y = StPlaneOf(v, S, i);
        double prevW = __shfl_up_sync(0xffffffffu, RC.v[kN - 1], 1), nextX = __shfl_down_sync(0xffffffffu, RC.v[0], 1);
        if (P.lane == 0) prevW = P.m0 > 0 ? R0[o - 1] * G0[o - 1] : 0.0;
        if (P.lane == 31) nextX = P.m0 + kN < P.RS ? R0[o + kN] * G0[o + kN] : 0.0;
        const int q = (i + P.j + 1) & 1;
        const Q2 sh = KShift(RC, prevW, nextX, q);
        Q2 nb;
#pragma unroll
        for (int x = 0; x < kN; x++)
            nb.v[x] = (rb.v[x] + StSum(S, Y, q, x, RP.v[x], RM.v[x], RJp.v[x], RJm.v[x], RC.v[x], sh.v[x])) * gb.v[x];
        if (P.valid)
        {
            SQ(X0 + o, RC);
            SQ(X1 + o, nb);
        }
        RM = RC;
        RC = RP;
    }
}

// One colour of a red-black sweep; kDot as SplitHalf's (nb_split.cu). r, idg, ec: this colour's halves, eo the other's.
template <int kDot>
__global__ void __launch_bounds__(kPairThreads, 3)
    k_stretched_half(LevelView v, const double *__restrict__ idg, const double *__restrict__ r,
                     const double *__restrict__ eo, double *__restrict__ ec, int colour, Reducer R, const int *it,
                     int baseEven, int baseOdd, int partSlot)
{
    PdlWait();
    PdlTrigger();
    const Blk blk = ThisBlk();
    double acc[3] = {0.0, 0.0, 0.0};
    QuadPos P = QuadStart<kN>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1))
    {
        if (!kDot) return;
        P.i1 = P.i0; // nothing to sweep; the block still adds its zero terms to the sums
    }
    const StRow S = StRowOf(v, P);
    const double *O = eo + P.off, *Rr = r + P.off, *G = idg + P.off;
    double *C = ec + P.off;
    Q2 oM{}, oC{};
    if (P.i0 < P.i1)
    {
        oM = LQ(O - P.PS);
        oC = LQ(O);
    }
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Q2 oP = LQ(O + o + P.PS), jp = LQ(O + o + P.RS), jm = LQ(O + o - P.RS);
        const Q2 rr = LQOnce(Rr + o), g = LQOnce(G + o);
        const StPlane Y = StPlaneOf(v, S, i);
        double prevW, nextX;
        Edges(P, oC, O + o, prevW, nextX);
        const int q = (i + P.j + colour) & 1;
        const Q2 sh = KShift(oC, prevW, nextX, q);
        Q2 nv;
#pragma unroll
        for (int x = 0; x < kN; x++)
            nv.v[x] = (rr.v[x] + StSum(S, Y, q, x, oP.v[x], oM.v[x], jp.v[x], jm.v[x], oC.v[x], sh.v[x])) * g.v[x];
        if (P.valid)
        {
            SQ(C + o, nv);
            if (kDot)
            {
#pragma unroll
                for (int x = 0; x < kN; x++)
                {
                    acc[0] += rr.v[x] * nv.v[x];
                    acc[1] += nv.v[x];
                    acc[2] += rr.v[x];
                }
            }
        }
        oM = oC;
        oC = oP;
    }
    if (kDot == 1) GridReduceB<3>(R, acc, partSlot, BlkId(blk), BlkCount(blk));
    else if (kDot == 2)
        GridReduceB<3>(R, acc, (*it & 1) ? baseOdd : baseEven, BlkId(blk), BlkCount(blk), 0, nullptr, partSlot);
}

// res = r - M e on the red cells after a sweep that ended black
__global__ void __launch_bounds__(kPairThreads, 3) k_stretched_residual(LevelView v, const uint8_t *__restrict__ du,
                                                                       const double *__restrict__ r,
                                                                       const double *__restrict__ e,
                                                                       double *__restrict__ res)
{
    PdlWait();
    PdlTrigger();
    const Blk blk = ThisBlk();
    const QuadPos P = QuadStart<kN>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1)) return;
    const StRow S = StRowOf(v, P);
    const double *O = e + v.sHalf + P.off, *Xr = e + P.off, *Rr = r + P.off, *G = v.dg + P.off;
    const uint8_t *D = du + P.off;
    Q2 oM = LQ(O - P.PS), oC = LQ(O);
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Q2 oP = LQ(O + o + P.PS), jp = LQ(O + o + P.RS), jm = LQ(O + o - P.RS);
        const Q2 xc = LQ(Xr + o), rr = LQOnce(Rr + o), g = LQ(G + o);
        const unsigned d = LdB<kN>(D + o);
        const StPlane Y = StPlaneOf(v, S, i);
        double prevW, nextX;
        Edges(P, oC, O + o, prevW, nextX);
        const int q = (i + P.j) & 1;
        const Q2 sh = KShift(oC, prevW, nextX, q);
        Q2 out;
#pragma unroll
        for (int x = 0; x < kN; x++)
        {
            const double s = StSum(S, Y, q, x, oP.v[x], oM.v[x], jp.v[x], jm.v[x], oC.v[x], sh.v[x]);
            out.v[x] = (Byte(d, x) & 0x80u) ? rr.v[x] - (g.v[x] * xc.v[x] - s) : 0.0;
        }
        if (P.valid) SQ(res + P.off + o, out);
        oM = oC;
        oC = oP;
    }
}

// p_new = U (z - mean + beta p_old), q = M p_new, sum p_new.q (SplitPApply's, nb_split.cu)
template <bool kSingular>
__global__ void __launch_bounds__(kPairThreads, 2)
    k_stretched_papply(LevelView v, const uint8_t *__restrict__ du, const double *__restrict__ z, double *p0,
                       double *p1, double *__restrict__ q, Reducer R, const double *Sl, const int *it, int baseEven,
                       int baseOdd, int slotN, int slotPQ)
{
    PdlWait();
    PdlTrigger();
    const Blk blk = ThisBlk();
    const int iter = *it, par = iter & 1;
    const double *__restrict__ pIn = par ? p1 : p0;
    double *__restrict__ pOut = par ? p0 : p1;
    const int baseNew = par ? baseOdd : baseEven, baseOld = par ? baseEven : baseOdd;
    const double n = Sl[slotN];
    auto rzEff = [&](int base) { return kSingular ? Sl[base] - (Sl[base + 1] / n) * Sl[base + 2] : Sl[base]; };
    const double bt = iter == 0 ? 0.0 : rzEff(baseNew) / rzEff(baseOld);
    const double mean = kSingular ? Sl[baseNew + 1] / n : 0.0;
    const QuadPos P = QuadStart<kN>(v, blk);
    double acc[1] = {0.0};
    if (TileIdle(v, blk.x, P.i0, P.i1))
    {
        GridReduceB<1>(R, acc, slotPQ, BlkId(blk), BlkCount(blk)); // p and q stay zero on these cells
        return;
    }
    const StRow S = StRowOf(v, P);
    const long long hb = v.sHalf;
    auto pn = [&](long long base) {
        const Q2 zz = LQ(z + base), pv = LQ(pIn + base);
        Q2 out;
#pragma unroll
        for (int x = 0; x < kN; x++) out.v[x] = (zz.v[x] - mean) + bt * pv.v[x];
        if (kSingular)
        {
            const unsigned d = LdB<kN>(du + base);
#pragma unroll
            for (int x = 0; x < kN; x++) out.v[x] *= Unk<double>(Byte(d, x));
        }
        return out;
    };
    auto pn1 = [&](long long idx) {
        double x = (z[idx] - mean) + bt * pIn[idx];
        if (kSingular) x *= Unk<double>(du[idx]);
        return x;
    };
    const long long b0 = P.off, b1 = hb + P.off;
    Q2 M0 = pn(b0 - P.PS), M1 = pn(b1 - P.PS), C0 = pn(b0), C1 = pn(b1);
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Q2 P0 = pn(b0 + o + P.PS), P1 = pn(b1 + o + P.PS);
        const Q2 Jp0 = pn(b0 + o + P.RS), Jp1 = pn(b1 + o + P.RS), Jm0 = pn(b0 + o - P.RS), Jm1 = pn(b1 + o - P.RS);
        const Q2 g0 = LQ(v.dg + b0 + o), g1 = LQ(v.dg + b1 + o);
        const StPlane Y = StPlaneOf(v, S, i);
        const int q0 = (i + P.j) & 1, q1 = q0 ^ 1;
        double pw0 = __shfl_up_sync(0xffffffffu, C0.v[kN - 1], 1), nx0 = __shfl_down_sync(0xffffffffu, C0.v[0], 1);
        double pw1 = __shfl_up_sync(0xffffffffu, C1.v[kN - 1], 1), nx1 = __shfl_down_sync(0xffffffffu, C1.v[0], 1);
        if (P.lane == 0 && P.m0 > 0)
        {
            pw0 = pn1(b0 + o - 1);
            pw1 = pn1(b1 + o - 1);
        }
        if (P.lane == 31 && P.m0 + kN < P.RS)
        {
            nx0 = pn1(b0 + o + kN);
            nx1 = pn1(b1 + o + kN);
        }
        const Q2 sh1 = KShift(C1, pw1, nx1, q0), sh0 = KShift(C0, pw0, nx0, q1);
        Q2 Q0, Q1;
#pragma unroll
        for (int x = 0; x < kN; x++)
        {
            // off the unknowns the diagonal is zero: masked through it (an isolated unknown's sum is zero too)
            const double s0 = StSum(S, Y, q0, x, P1.v[x], M1.v[x], Jp1.v[x], Jm1.v[x], C1.v[x], sh1.v[x]);
            const double s1 = StSum(S, Y, q1, x, P0.v[x], M0.v[x], Jp0.v[x], Jm0.v[x], C0.v[x], sh0.v[x]);
            Q0.v[x] = g0.v[x] != 0.0 ? g0.v[x] * C0.v[x] - s0 : 0.0;
            Q1.v[x] = g1.v[x] != 0.0 ? g1.v[x] * C1.v[x] - s1 : 0.0;
        }
        if (P.valid)
        {
            SQ(pOut + b0 + o, C0);
            SQ(pOut + b1 + o, C1);
            SQ(q + b0 + o, Q0);
            SQ(q + b1 + o, Q1);
#pragma unroll
            for (int x = 0; x < kN; x++) acc[0] += C0.v[x] * Q0.v[x] + C1.v[x] * Q1.v[x];
        }
        M0 = C0;
        M1 = C1;
        C0 = P0;
        C1 = P1;
    }
    GridReduceB<1>(R, acc, slotPQ, BlkId(blk), BlkCount(blk));
}

// ---- launchers ----
void LaunchStretchedFirst(const LevelView &v, const double *r, double *e, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(k_stretched_first, QuadGrid<kN>(v, Occ<k_stretched_first>()), kPairThreads, 0, st, v, r, e);
}

template <int kDot>
static void HalfOn(const LevelView &v, const double *r, double *e, int c, const Reducer &R, const int *it, int baseEven,
                   int baseOdd, int partSlot, cudaStream_t st)
{
    const long long h = v.sHalf;
    NB_COUNT_LAUNCH();
    const dim3 grid = QuadGrid<kN>(v, Occ<k_stretched_half<kDot>>());
    LaunchPdl(k_stretched_half<kDot>, kDot ? SumGrid(R, grid) : grid, kPairThreads, 0, st, v, v.idg + c * h, r + c * h,
              (const double *)(e + (c ^ 1) * h), e + c * h, c, R, it, baseEven, baseOdd, partSlot);
}

void LaunchStretchedHalf(const LevelView &v, const double *r, double *e, int colour, cudaStream_t st)
{
    HalfOn<0>(v, r, e, colour, Reducer{}, nullptr, 0, 0, 0, st);
}

void LaunchStretchedHalfDot(const LevelView &v, const double *r, double *e, int colour, bool last, const Reducer &R,
                            const int *it, int baseEven, int baseOdd, int partSlot, cudaStream_t st)
{
    if (last) HalfOn<2>(v, r, e, colour, R, it, baseEven, baseOdd, partSlot, st);
    else HalfOn<1>(v, r, e, colour, R, it, baseEven, baseOdd, partSlot, st);
}

void LaunchStretchedResidual(const LevelView &v, const uint8_t *du, const double *r, const double *e, double *res,
                             cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(k_stretched_residual, QuadGrid<kN>(v, Occ<k_stretched_residual>()), kPairThreads, 0, st, v, du, r, e,
              res);
}

void LaunchStretchedPApply(const LevelView &v, const uint8_t *du, const double *z, double *p0, double *p1, double *q,
                           const Reducer &R, const double *S, const int *it, int baseEven, int baseOdd, int slotN,
                           int singular, int slotPQ, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if (singular)
        LaunchPdl(k_stretched_papply<true>, SumGrid(R, QuadGrid<kN>(v, Occ<k_stretched_papply<true>>())), kPairThreads, 0,
                  st, v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, slotPQ);
    else
        LaunchPdl(k_stretched_papply<false>, SumGrid(R, QuadGrid<kN>(v, Occ<k_stretched_papply<false>>())), kPairThreads, 0,
                  st, v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, slotPQ);
}

// the kernels' occupancy, read outside any stream capture
void PrepareStretchedKernels()
{
    (void)Occ<k_stretched_first>();
    (void)Occ<k_stretched_half<0>>();
    (void)Occ<k_stretched_half<1>>();
    (void)Occ<k_stretched_half<2>>();
    (void)Occ<k_stretched_residual>();
    (void)Occ<k_stretched_papply<true>>();
    (void)Occ<k_stretched_papply<false>>();
}

} // namespace nb
