// Multigrid and PCG kernels for uniform 3D levels in the colour-split layout, built so that each red-black half-sweep
// moves only the bytes the algorithm needs: T = float for the inner solve of the mixed-precision form, double for the
// plain FP64 form.
//
// Colour-split layout. Cell (i, j, k) has colour c = (i + j + k) & 1 and sits at c*H + i*PS + j*RS + (k >> 1) of a
// level vector: each colour is an Ny x Nx x RS array whose rows hold that colour's cells (RS = (Nz+1)/2 rounded up
// to 4, the padding kept at zero; with Nz odd the rows of one colour hold a cell less, its element counts as padding).
// In row (i, j) the cell of colour c at element m is k = 2m + q with q = (i + j + c) & 1, and its six neighbours all have
// the other colour:
//   (i +- 1, j, m), (i, j +- 1, m), (i, j, m) and (i, j, m + (q ? 1 : -1)).
// A half-sweep of colour c therefore reads the other colour, r and the diagonal bytes of colour c, and writes
// colour c: half of every array, where a cell-pair sweep reads and writes both colours.
//
// Quads. Thread t of a launch takes the 16 bytes of elements N t .. N t + N - 1 of a plane of one colour (N = 4 floats
// or 2 doubles; RS is a multiple of 4, so a quad never crosses a row) and marches along i over up to kQuadMaxS planes,
// keeping planes i-1, i, i+1 in registers. The j neighbours are the quads RS elements away; the element across the
// quad's edge comes from the neighbouring lane (a shuffle; lanes 0 and 31 load it). Two doubles a thread keep the FP64
// kernels at the FP32 ones' register counts and loads in flight. FP64 at 256^3 (B200): these kernels took the plain
// form's step from 25.0 ms (one thread per cell, a code and a neighbour mask per cell; the bytes of its 12 iterations at
// 0.24 of the measured copy bandwidth) to 9.8 ms (0.62).
//
// Every vector is zero off the unknowns (and on the padding), so the neighbour sum runs over all six neighbours. The
// levels are uniform (a stretched level's sweeps are in nb_stretched.cu, the transfers here): the coefficient is gamma
// everywhere and the diagonal is gamma/2 times the unit count in the level's byte array (0x80 | units, 0 off the
// unknowns), divided through a 32-entry reciprocal table.
//
// The V-cycle on these levels (nb_solver.cu, VCycleSplit) uses two facts of red-black Gauss-Seidel:
// - after a black half-sweep the black residual is zero (each black equation was just solved), so the residual and
//   its restriction run over the red cells only;
// - a black half-sweep does not read the black values it replaces, so the prolonged coarse correction is added to
//   the red cells only before the post-smoothing, which starts black.
#include "nb_quad.cuh"

namespace nb
{

bool SplitLevelShape(const LevelView &v) { return v.dim == 3 && v.Nx >= 3 && v.Ny >= 3 && v.Nz >= 3; }

// ---------------------------------------------------------------------------------------------------------------
// smoothing
// ---------------------------------------------------------------------------------------------------------------

// The first red-black sweep from a zero iterate on a uniform level, one launch: red e = r / diag, then black
// e = (r + gamma * sum of the red neighbours) / diag with the red neighbours formed from r and the bytes. A thread
// owns one quad position and writes the red and the black quad there.
template <typename T>
__device__ __forceinline__ void SplitFirst(const LevelView &v, const uint8_t *__restrict__ du,
                                           const T *__restrict__ r, T *__restrict__ e, const Blk &blk)
{
    constexpr int N = kQ<T>;
    __shared__ T inv[32];
    FillInv<T>(inv, v.gamma);
    const QuadPos P = QuadStart<N>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1)) return;
    const T g = (T)v.gamma;
    const long long hb = v.sHalf;
    const T *R0 = r + P.off, *R1 = r + hb + P.off;
    const uint8_t *D0 = du + P.off, *D1 = du + hb + P.off;
    T *X0 = e + P.off, *X1 = e + hb + P.off;
    auto red = [&](long long o) {
        Quad<T> a = LQ(R0 + o);
        const unsigned d = LdB<N>(D0 + o);
#pragma unroll
        for (int x = 0; x < N; x++) a.v[x] *= inv[Byte(d, x) & 0x7Fu];
        return a;
    };
    auto red1 = [&](long long o) { return R0[o] * inv[D0[o] & 0x7Fu]; };
    Quad<T> RM = red(-P.PS), RC = red(0);
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Quad<T> RP = red(o + P.PS), RJp = red(o + P.RS), RJm = red(o - P.RS);
        const Quad<T> rb = LQOnce(R1 + o);
        const unsigned db = LdBOnce<N>(D1 + o);
        T prevW = __shfl_up_sync(0xffffffffu, RC.v[N - 1], 1), nextX = __shfl_down_sync(0xffffffffu, RC.v[0], 1);
        if (P.lane == 0) prevW = P.m0 > 0 ? red1(o - 1) : (T)0;
        if (P.lane == 31) nextX = P.m0 + N < P.RS ? red1(o + N) : (T)0;
        const Quad<T> sh = KShift(RC, prevW, nextX, (i + P.j + 1) & 1);
        Quad<T> nb;
#pragma unroll
        for (int x = 0; x < N; x++)
        {
            const T s = ((RP.v[x] + RM.v[x]) + (RJp.v[x] + RJm.v[x])) + (RC.v[x] + sh.v[x]);
            nb.v[x] = (rb.v[x] + g * s) * inv[Byte(db, x) & 0x7Fu];
        }
        if (P.valid)
        {
            SQ(X0 + o, RC);
            SQ(X1 + o, nb);
        }
        RM = RC;
        RC = RP;
    }
}

template <typename T>
__global__ void __launch_bounds__(kPairThreads) k_split_first(LevelView v, const uint8_t *__restrict__ du,
                                                              const T *__restrict__ r, T *__restrict__ e)
{
    PdlWait();
    PdlTrigger();
    SplitFirst<T>(v, du, r, e, ThisBlk());
}

// One colour of a red-black sweep: e_c = (r_c + gamma * sum of the other colour's six neighbours) / diag_c.
// kDot 1: (sum r.e, sum e, sum r) of this colour into out[partSlot..]; kDot 2: the same plus the totals already in
// out[partSlot..], into the scalar block of the iteration's parity (the CG's r.z, sum z, sum r of the V-cycle's z).
// du, r: this colour's halves; eo, ec: the other colour's and this colour's halves of e (disjoint).
template <typename T, int kDot>
__device__ __forceinline__ void SplitHalf(const LevelView &v, const uint8_t *__restrict__ du,
                                          const T *__restrict__ r, const T *__restrict__ eo,
                                          T *__restrict__ ec, int colour, const Reducer &R, const int *it,
                                          int baseEven, int baseOdd, int partSlot, const Blk &blk)
{
    constexpr int N = kQ<T>;
    T facc[3] = {(T)0, (T)0, (T)0}; // a thread's terms in T, the block and grid sums in FP64
    __shared__ T inv[32];
    FillInv<T>(inv, v.gamma);
    QuadPos P = QuadStart<N>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1))
    {
        if (!kDot) return;
        P.i1 = P.i0; // nothing to sweep; the block still adds its zero terms to the sums
    }
    const T g = (T)v.gamma;
    const T *O = eo + P.off;
    const T *Rr = r + P.off;
    const uint8_t *D = du + P.off;
    T *C = ec + P.off;
    // one plane: the six other-colour neighbours, r and the bytes given, the new values stored (and summed)
    auto plane = [&](int i, long long o, const Quad<T> &oM, const Quad<T> &oC, const Quad<T> &oP, const Quad<T> &jp,
                     const Quad<T> &jm, const Quad<T> &rr, unsigned d) {
        T prevW, nextX;
        Edges(P, oC, O + o, prevW, nextX);
        const Quad<T> sh = KShift(oC, prevW, nextX, (i + P.j + colour) & 1);
        Quad<T> nv;
#pragma unroll
        for (int x = 0; x < N; x++)
        {
            const T s = ((oP.v[x] + oM.v[x]) + (jp.v[x] + jm.v[x])) + (oC.v[x] + sh.v[x]);
            nv.v[x] = (rr.v[x] + g * s) * inv[Byte(d, x) & 0x7Fu];
        }
        if (P.valid)
        {
            SQ(C + o, nv);
            if (kDot)
            {
#pragma unroll
                for (int x = 0; x < N; x++)
                {
                    facc[0] += rr.v[x] * nv.v[x];
                    facc[1] += nv.v[x];
                    facc[2] += rr.v[x];
                }
            }
        }
    };
    // two planes per trip: all the streamed values of both (the other colour up to two planes ahead, the j rows,
    // r and the bytes) are loaded before either is computed, twice the loads in flight of a plane-by-plane march
    Quad<T> oM{}, oC{};
    if (P.i0 < P.i1)
    {
        oM = LQ(O - P.PS);
        oC = LQ(O);
    }
    long long o = 0;
    for (int i = P.i0; i < P.i1; i += 2, o += 2 * P.PS)
    {
        const bool two = i + 1 < P.i1;
        const Quad<T> oP = LQ(O + o + P.PS);
        const Quad<T> oPP = two ? LQ(O + o + 2 * P.PS) : Quad<T>{};
        const Quad<T> r0 = LQOnce(Rr + o), r1 = two ? LQOnce(Rr + o + P.PS) : Quad<T>{};
        const unsigned d0 = LdBOnce<N>(D + o), d1 = two ? LdBOnce<N>(D + o + P.PS) : 0u;
        const Quad<T> jp0 = LQ(O + o + P.RS), jm0 = LQ(O + o - P.RS);
        const Quad<T> jp1 = two ? LQ(O + o + P.PS + P.RS) : Quad<T>{}, jm1 = two ? LQ(O + o + P.PS - P.RS) : Quad<T>{};
        plane(i, o, oM, oC, oP, jp0, jm0, r0, d0);
        if (two) plane(i + 1, o + P.PS, oC, oP, oPP, jp1, jm1, r1, d1);
        oM = oP;
        oC = oPP;
    }
    if (kDot == 1)
    {
        double acc[3] = {facc[0], facc[1], facc[2]};
        GridReduceB<3>(R, acc, partSlot, BlkId(blk), BlkCount(blk));
    }
    else if (kDot == 2)
    {
        double acc[3] = {facc[0], facc[1], facc[2]};
        GridReduceB<3>(R, acc, (*it & 1) ? baseOdd : baseEven, BlkId(blk), BlkCount(blk), 0, nullptr, partSlot);
    }
}

// 4 resident blocks (64 registers): the two-plane march measured 12% faster there than at 3 (73 registers)
template <typename T, int kDot>
__global__ void __launch_bounds__(kPairThreads, 4)
    k_split_half(LevelView v, const uint8_t *__restrict__ du, const T *__restrict__ r,
                 const T *__restrict__ eo, T *__restrict__ ec, int colour, Reducer R, const int *it,
                 int baseEven, int baseOdd, int partSlot)
{
    PdlWait();
    PdlTrigger();
    SplitHalf<T, kDot>(v, du, r, eo, ec, colour, R, it, baseEven, baseOdd, partSlot, ThisBlk());
}

// the arguments of k_split_half for colour c: its halves of du and r, the other colour's and its own halves of e
#define NB_SPLIT_HALF_ARGS(c)                                                                                      \
    v, du + (long long)(c) * v.sHalf, r + (long long)(c) * v.sHalf, e + (long long)((c) ^ 1) * v.sHalf,               \
        e + (long long)(c) * v.sHalf, (c)

template <typename T>
void LaunchSplitFirst(const LevelView &v, const uint8_t *du, const T *r, T *e, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8)
        if (v.stretched) return LaunchStretchedFirst(v, r, e, st);
    NB_COUNT_LAUNCH();
    LaunchPdl(k_split_first<T>, QuadGrid<kQ<T>>(v, Occ<k_split_first<T>>()), kPairThreads, 0, st, v, du, r, e);
}

template <typename T>
void LaunchSplitHalf(const LevelView &v, const uint8_t *du, const T *r, T *e, int colour, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8)
        if (v.stretched) return LaunchStretchedHalf(v, r, e, colour, st);
    NB_COUNT_LAUNCH();
    LaunchPdl(k_split_half<T, 0>, QuadGrid<kQ<T>>(v, Occ<k_split_half<T, 0>>()), kPairThreads, 0, st,
              NB_SPLIT_HALF_ARGS(colour), Reducer{}, (const int *)nullptr, 0, 0, 0);
}

template <typename T>
void LaunchSplitHalfDot(const LevelView &v, const uint8_t *du, const T *r, T *e, int colour, bool last,
                        const Reducer &R, const int *it, int baseEven, int baseOdd, int partSlot, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8)
        if (v.stretched) return LaunchStretchedHalfDot(v, r, e, colour, last, R, it, baseEven, baseOdd, partSlot, st);
    NB_COUNT_LAUNCH();
    if (last)
        LaunchPdl(k_split_half<T, 2>, SumGrid(R, QuadGrid<kQ<T>>(v, Occ<k_split_half<T, 2>>())), kPairThreads, 0, st,
                  NB_SPLIT_HALF_ARGS(colour), R, it, baseEven, baseOdd, partSlot);
    else
        LaunchPdl(k_split_half<T, 1>, SumGrid(R, QuadGrid<kQ<T>>(v, Occ<k_split_half<T, 1>>())), kPairThreads, 0, st,
                  NB_SPLIT_HALF_ARGS(colour), R, it, baseEven, baseOdd, partSlot);
}
#undef NB_SPLIT_HALF_ARGS

// res = r - M e on the red cells (colour 0), into the first half of `res`; the black residual after a black
// half-sweep is zero.
template <typename T>
__device__ __forceinline__ void SplitResidual(const LevelView &v, const uint8_t *__restrict__ du,
                                              const T *__restrict__ r, const T *__restrict__ e,
                                              T *__restrict__ res, const Blk &blk)
{
    constexpr int N = kQ<T>;
    const QuadPos P = QuadStart<N>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1)) return;
    const T g = (T)v.gamma, hg = (T)0.5 * (T)v.gamma;
    const T *O = e + v.sHalf + P.off;
    const T *Xr = e + P.off;
    const T *Rr = r + P.off;
    const uint8_t *D = du + P.off;
    T *Out = res + P.off;
    auto plane = [&](int i, long long o, const Quad<T> &oM, const Quad<T> &oC, const Quad<T> &oP, const Quad<T> &jp,
                     const Quad<T> &jm, const Quad<T> &xc, const Quad<T> &rr, unsigned d) {
        T prevW, nextX;
        Edges(P, oC, O + o, prevW, nextX);
        const Quad<T> sh = KShift(oC, prevW, nextX, (i + P.j) & 1);
        Quad<T> out;
#pragma unroll
        for (int x = 0; x < N; x++)
        {
            const unsigned b = Byte(d, x);
            const T s = ((oP.v[x] + oM.v[x]) + (jp.v[x] + jm.v[x])) + (oC.v[x] + sh.v[x]);
            out.v[x] = (b & 0x80u) ? rr.v[x] - (hg * (T)(b & 0x7Fu) * xc.v[x] - g * s) : (T)0;
        }
        if (P.valid) SQ(Out + o, out);
    };
    // two planes per trip, all their streamed values loaded first (as in the half-sweep)
    Quad<T> oM = LQ(O - P.PS), oC = LQ(O);
    long long o = 0;
    for (int i = P.i0; i < P.i1; i += 2, o += 2 * P.PS)
    {
        const bool two = i + 1 < P.i1;
        const Quad<T> oP = LQ(O + o + P.PS), oPP = two ? LQ(O + o + 2 * P.PS) : Quad<T>{};
        const Quad<T> jp0 = LQ(O + o + P.RS), jm0 = LQ(O + o - P.RS);
        const Quad<T> jp1 = two ? LQ(O + o + P.PS + P.RS) : Quad<T>{}, jm1 = two ? LQ(O + o + P.PS - P.RS) : Quad<T>{};
        const Quad<T> x0 = LQ(Xr + o), r0 = LQOnce(Rr + o), x1 = two ? LQ(Xr + o + P.PS) : Quad<T>{},
                      r1 = two ? LQOnce(Rr + o + P.PS) : Quad<T>{};
        const unsigned d0 = LdBOnce<N>(D + o), d1 = two ? LdBOnce<N>(D + o + P.PS) : 0u;
        plane(i, o, oM, oC, oP, jp0, jm0, x0, r0, d0);
        if (two) plane(i + 1, o + P.PS, oC, oP, oPP, jp1, jm1, x1, r1, d1);
        oM = oP;
        oC = oPP;
    }
}

template <typename T>
__global__ void __launch_bounds__(kPairThreads, sizeof(T) == 8 ? 3 : 4)
    k_split_residual(LevelView v, const uint8_t *__restrict__ du, const T *__restrict__ r, const T *__restrict__ e,
                     T *__restrict__ res)
{
    PdlWait();
    PdlTrigger();
    SplitResidual<T>(v, du, r, e, res, ThisBlk());
}

template <typename T>
void LaunchSplitResidual(const LevelView &v, const uint8_t *du, const T *r, const T *e, T *res, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8)
        if (v.stretched) return LaunchStretchedResidual(v, du, r, e, res, st);
    NB_COUNT_LAUNCH();
    LaunchPdl(k_split_residual<T>, QuadGrid<kQ<T>>(v, Occ<k_split_residual<T>>()), kPairThreads, 0, st, v, du, r, e,
              res);
}

// ---------------------------------------------------------------------------------------------------------------
// transfers between a split level and the next coarser level (either layout): the operators of k_prolong and
// k_restrict on the red cells
// ---------------------------------------------------------------------------------------------------------------
// Per red fine cell (colour-split, red half only): 0x80 for an unknown, plus in the low six bits the weight (in 1/64)
// that the Neumann-aware prolongation moves from the cell's SOLID coarse contributors onto its parent.

// e_f += P e_c on the red fine unknowns. Fine k = 2m + q (q = (a + b) & 1) lies between coarse k-cells m and m+1
// with weights (3/4, 1/4) for q = 0 and (1/4, 3/4) for q = 1; its parent is m + q. Fine row 2B-1 mixes coarse rows
// B (3/4) and B-1 (1/4), row 2B rows B and B+1; planes the same way.
//
// A thread owns coarse row B and the fine quad m0 .. m0+3 of fine rows 2B-1 and 2B, and marches along the coarse
// planes A: per coarse plane it interpolates three coarse rows across j once (k-cells m0 .. m0+4), and with the
// neighbouring planes' rows (kept in registers) serves the four fine quads of fine planes 2A-1, 2A and rows 2B-1,
// 2B, whose red values and bytes it loads together.

// coarse k-cells m0 .. m0+N of coarse row (A, B), N = kQ<T>
template <typename T>
__device__ __forceinline__ void CoarseRowK(const LevelView &cv, const T *__restrict__ ec, int A, int B, int m0,
                                           T c[kQ<T> + 1])
{
    constexpr int N = kQ<T>;
    const int Dmax = cv.Nz - 1;
    if (cv.sRS && m0 + N <= Dmax)
    {
        // a colour-split coarse level: the even k-cells m0, m0+2, .. are elements m0/2, m0/2+1, .. of colour
        // (A+B) & 1, the odd ones the same elements of the other (m0 is a multiple of N)
        const int ce = (A + B) & 1;
        const T *rb = ec + (long long)A * cv.sPS + (long long)B * cv.sRS + (m0 >> 1);
        if constexpr (N == 4)
        {
            const float2 ev = *reinterpret_cast<const float2 *>(rb + ce * cv.sHalf);
            const float2 od = *reinterpret_cast<const float2 *>(rb + (ce ^ 1) * cv.sHalf);
            c[0] = ev.x;
            c[1] = od.x;
            c[2] = ev.y;
            c[3] = od.y;
            c[4] = rb[ce * cv.sHalf + 2];
        }
        else
        {
            c[0] = rb[ce * cv.sHalf];
            c[1] = rb[(ce ^ 1) * cv.sHalf];
            c[2] = rb[ce * cv.sHalf + 1];
        }
        return;
    }
#pragma unroll
    for (int t = 0; t <= N; t++) c[t] = ec[VecIdx(cv, A, B, min(m0 + t, Dmax))]; // past the row: masked cells only
}

// the coarse plane's rows interpolated across j for fine rows 2B-1 (y0) and 2B (y1), and row B itself (par); one: row B
// has a single fine row (x groups), which takes it whole
template <typename T>
__device__ __forceinline__ void CoarsePlaneRows(const LevelView &cv, const T *__restrict__ ec, int A, int B, int m0,
                                                bool one, T y0[kQ<T> + 1], T y1[kQ<T> + 1], T par[kQ<T> + 1])
{
    T cm[kQ<T> + 1], cp[kQ<T> + 1];
    CoarseRowK<T>(cv, ec, A, B, m0, par);
    CoarseRowK<T>(cv, ec, A, B - 1, m0, cm);
    CoarseRowK<T>(cv, ec, A, B + 1, m0, cp);
#pragma unroll
    for (int t = 0; t <= kQ<T>; t++)
    {
        y0[t] = one ? par[t] : (T)0.75 * par[t] + (T)0.25 * cm[t];
        y1[t] = (T)0.75 * par[t] + (T)0.25 * cp[t];
    }
}

// kX: the coarsening keeps some x cells whole (LevelView::xr: row B's first fine row, and whether it has a second)
template <typename T, bool kX>
__device__ __forceinline__ void SplitProlong(const LevelView &fv, const LevelView &cv,
                                             const uint8_t *__restrict__ pext, const T *__restrict__ ec,
                                             T *__restrict__ ef, const Blk &blk)
{
    constexpr int N = kQ<T>;
    constexpr unsigned kUnkMask = N == 4 ? 0x80808080u : 0x8080u;
    const int Q = fv.sRS / N, nrow = cv.Nx - 2, nq = nrow * Q;
    int t = blk.x * kPairThreads + threadIdx.x;
    const bool valid = t < nq;
    if (!valid) t = nq - 1;
    const int B = 1 + t / Q, m0 = N * (t - (B - 1) * Q);
    const int S = (cv.Ny - 2 + blk.gy - 1) / blk.gy;
    const int A0 = min(1 + blk.y * S, cv.Ny - 1), A1 = min(A0 + S, cv.Ny - 1);
    if (!valid || A0 >= A1) return;
    // a block whose fine rows hold no unknown on its planes adds nothing (the air of a tank)
    {
        const int t0 = blk.x * kPairThreads, B0 = 1 + t0 / Q, B1 = 1 + min(t0 + kPairThreads, nq) / Q;
        const int f0 = kX ? (fv.xr[B0] & 0x7FFF) : 2 * B0 - 1;
        const int f1 = kX ? (fv.xr[min(B1, nrow)] & 0x7FFF) + 1 : 2 * min(B1, nrow);
        if (RowsIdle<N * kPairThreads>(fv, f0, min(f1, fv.Nx - 1), 2 * A0 - 1, 2 * A1 - 1)) return;
    }
    const int xg = kX ? fv.xr[B] : 0;
    const bool one = kX && !((xg >> 15) & 1);
    const int fb0 = kX ? (xg & 0x7FFF) : 2 * B - 1, fb1 = one ? fb0 : fb0 + 1;
    T yM0[N + 1], yM1[N + 1], yC0[N + 1], yC1[N + 1], pC[N + 1], pD[N + 1];
    CoarsePlaneRows<T>(cv, ec, A0 - 1, B, m0, one, yM0, yM1, pD);
    CoarsePlaneRows<T>(cv, ec, A0, B, m0, one, yC0, yC1, pC);
    for (int A = A0; A < A1; A++)
    {
        T yP0[N + 1], yP1[N + 1], pP[N + 1];
        // the four fine quads and their bytes, loaded with the coarse plane's rows: behind the stores of the first two,
        // the last two waited for memory once more (258^3 level, FP32, B200: 31.8 -> 25.0 us)
        Quad<T> ev[2][2];
        unsigned wv[2][2];
#pragma unroll
        for (int h = 0; h < 2; h++)
        {
            const long long o0 = (long long)min(2 * A - 1 + h, fv.Ny - 1) * fv.sPS + (long long)fb0 * fv.sRS + m0;
            const long long o1 = one ? o0 : (long long)min(fb1, fv.Nx - 1) * fv.sRS - (long long)fb0 * fv.sRS + o0;
            wv[h][0] = LdB<N>(pext + o0);
            wv[h][1] = LdB<N>(pext + o1);
            ev[h][0] = LQ(ef + o0);
            ev[h][1] = LQ(ef + o1);
            if (one) wv[h][1] = 0u;
        }
        CoarsePlaneRows<T>(cv, ec, A + 1, B, m0, one, yP0, yP1, pP);
        // fine planes 2A-1 (with coarse plane A-1) and 2A (with A+1), rows 2B-1 and 2B
#pragma unroll
        for (int h = 0; h < 2; h++)
        {
            const int fa = 2 * A - 1 + h;
            const long long o0 = (long long)fa * fv.sPS + (long long)fb0 * fv.sRS + m0, o1 = o0 + fv.sRS;
            const unsigned w0 = wv[h][0], w1 = wv[h][1];
            Quad<T> &e0 = ev[h][0], &e1 = ev[h][1];
            const T *yo0 = h ? yP0 : yM0, *yo1 = h ? yP1 : yM1;
#pragma unroll
            for (int rI = 0; rI < 2; rI++)
            {
                const unsigned w = rI ? w1 : w0;
                if (!(w & kUnkMask)) continue;
                const int q = (fa + (rI ? fb1 : fb0)) & 1;
                T z[N + 1];
#pragma unroll
                for (int k = 0; k <= N; k++)
                    z[k] = rI ? (T)0.75 * yC1[k] + (T)0.25 * yo1[k] : (T)0.75 * yC0[k] + (T)0.25 * yo0[k];
                Quad<T> &er = rI ? e1 : e0;
#pragma unroll
                for (int x = 0; x < N; x++)
                {
                    const unsigned px = Byte(w, x);
                    if (!(px & 0x80u)) continue;
                    const T lohi = q ? (T)0.25 * z[x] + (T)0.75 * z[x + 1] : (T)0.75 * z[x] + (T)0.25 * z[x + 1];
                    er.v[x] += lohi + (T)(px & 0x3Fu) * (T)(1.0 / 64.0) * (q ? pC[x + 1] : pC[x]);
                }
                SQ(ef + (rI ? o1 : o0), er);
            }
        }
#pragma unroll
        for (int k = 0; k <= N; k++)
        {
            yM0[k] = yC0[k];
            yM1[k] = yC1[k];
            yC0[k] = yP0[k];
            yC1[k] = yP1[k];
            pC[k] = pP[k];
        }
    }
}

// 2 resident blocks: at 3 (80 registers) 136 bytes are spilled and the 258^3 level takes 28.1 us, here 25.0
template <typename T, bool kX>
__global__ void __launch_bounds__(kPairThreads, 2) k_split_prolong(LevelView fv, LevelView cv,
                                                                const uint8_t *__restrict__ pext,
                                                                const T *__restrict__ ec, T *__restrict__ ef)
{
    PdlWait();
    PdlTrigger();
    SplitProlong<T, kX>(fv, cv, pext, ec, ef, ThisBlk());
}

// The grid of k_split_prolong: threads over (coarse row, fine quad), grid.y chunks of coarse planes sized like
// QuadGrid's (the longest march with a full last wave).
template <int N = 4> inline dim3 ProlongGridS(const LevelView &fine, const LevelView &coarse, int S)
{
    const long long nq = (long long)(coarse.Nx - 2) * (fine.sRS / N), perPlane = (nq + kPairThreads - 1) / kPairThreads;
    const long long planes = coarse.Ny - 2 > 0 ? coarse.Ny - 2 : 1;
    return dim3((unsigned)perPlane, (unsigned)((planes + S - 1) / S));
}

template <int N> inline dim3 ProlongGrid(const LevelView &fine, const LevelView &coarse, int resident)
{
    const long long nq = (long long)(coarse.Nx - 2) * (fine.sRS / N), perPlane = (nq + kPairThreads - 1) / kPairThreads;
    const long long planes = coarse.Ny - 2 > 0 ? coarse.Ny - 2 : 1;
    const long long bestS = BestMarch(perPlane, planes, (long long)SmCount() * (resident > 0 ? resident : 1));
    return dim3((unsigned)perPlane, (unsigned)((planes + bestS - 1) / bestS));
}

template <typename T>
void LaunchSplitProlong(const LevelView &fine, const LevelView &coarse, const uint8_t *pext, const T *eCoarse,
                        T *eFine, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if constexpr (sizeof(T) == 8) // stretched grids run on this layout in FP64
        if (fine.xr)
        {
            const int occ = Occ<k_split_prolong<T, true>>();
            LaunchPdl(k_split_prolong<T, true>, ProlongGrid<kQ<T>>(fine, coarse, occ), kPairThreads, 0, st, fine,
                      coarse, pext, eCoarse, eFine);
            return;
        }
    const int occ = Occ<k_split_prolong<T, false>>();
    LaunchPdl(k_split_prolong<T, false>, ProlongGrid<kQ<T>>(fine, coarse, occ), kPairThreads, 0, st, fine, coarse,
              pext, eCoarse, eFine);
}

// r_c = R res_f = P^T res_f at the coarse unknowns, from the red fine residual. A thread owns N = 4 (FP64: 2) consecutive
// coarse cells K0 .. K0+N-1 (K0 = 1 + N t) of coarse row J (one flat index over (J, t)) and marches along I: fine planes
// 2I-2 .. 2I+1 enter as their (j, k)-weighted 4x4 sums T(a), each kept for the next coarse plane; the red children's
// moved weights enter as X(a). In fine row (a, b) the red cells among k = 2K-2 .. 2K+1 are elements K-1 and K, at
// k = 2K-2+q and 2K+q (q = (a + b) & 1), and the red child of coarse K is element K - q; the N + 1 elements
// K0-1 .. K0+N-1 of a row are one aligned quad and one more.
// The fine rows coarse row J gathers from and their weights: 2J-2 .. 2J+1, or with x groups (kX) those of
// LevelView::xr; rows 1 and 2 are J's children (row 2 only with two).
template <typename T, bool kX> struct RowTaps
{
    int b[4];
    T w[4];
    bool two;
};
template <typename T, bool kX> __device__ __forceinline__ RowTaps<T, kX> TapsOf(const LevelView &fv, int J)
{
    RowTaps<T, kX> t;
    if constexpr (kX) XrTaps<T>(fv.xr[J], t.b, t.w, t.two);
    else
    {
        t.two = true;
#pragma unroll
        for (int dj = 0; dj < 4; dj++)
        {
            t.b[dj] = 2 * J - 2 + dj;
            t.w[dj] = dj == 0 || dj == 3 ? (T)0.25 : (T)0.75;
        }
    }
    return t;
}

// What one fine plane gives: four rows of N + 1 elements and the children's transfer bytes, all loaded before any is
// used. With a branch around each row past the level's edge the rows were loaded one after the other, each waiting for
// the last (258^3 level, FP32, B200: 31.7 -> 21.9 us); now such rows and planes read the ring, which is zero.
template <typename T> struct RestrictLoads
{
    Quad<T> r[4];
    T rN[4];
    unsigned w[2], wN[2];
};
template <typename T, bool kX>
__device__ __forceinline__ RestrictLoads<T> LoadRestrict(const LevelView &fv, const uint8_t *__restrict__ pext,
                                                         const T *__restrict__ res, int a, const RowTaps<T, kX> &J,
                                                         int K0, bool more)
{
    constexpr int N = kQ<T>;
    RestrictLoads<T> l;
    const long long base = (long long)min(a, fv.Ny - 1) * fv.sPS + (K0 - 1);
#pragma unroll
    for (int dj = 0; dj < 4; dj++)
    {
        const long long row = base + (long long)min(J.b[dj], fv.Nx - 1) * fv.sRS;
        l.r[dj] = LQ(res + row);
        l.rN[dj] = more ? res[row + N] : (T)0;
        if (dj == 1 || dj == 2)
        {
            l.w[dj - 1] = LdB<N>(pext + row);
            l.wN[dj - 1] = more ? pext[row + N] : 0u;
        }
    }
    return l;
}

template <typename T, bool kX>
__device__ __forceinline__ void SplitRestrictPlane(const RestrictLoads<T> &l, int a, const RowTaps<T, kX> &J,
                                                   T (&Tw)[kQ<T>], T (&X)[kQ<T>])
{
    constexpr int N = kQ<T>;
#pragma unroll
    for (int x = 0; x < N; x++) Tw[x] = X[x] = (T)0;
#pragma unroll
    for (int dj = 0; dj < 4; dj++)
    {
        const int q = (a + J.b[dj]) & 1;
        const bool none = kX && J.w[dj] == (T)0; // a tap that is not there
        T R[N + 1];
#pragma unroll
        for (int x = 0; x < N; x++) R[x] = none ? (T)0 : l.r[dj].v[x];
        R[N] = none ? (T)0 : l.rN[dj];
#pragma unroll
        for (int x = 0; x < N; x++)
            Tw[x] += J.w[dj] * (q ? (T)0.75 * R[x] + (T)0.25 * R[x + 1] : (T)0.25 * R[x] + (T)0.75 * R[x + 1]);
        if (dj == 1 || (dj == 2 && J.two))
        {
#pragma unroll
            for (int x = 0; x < N; x++)
            {
                // the red child of coarse K0 + x is element K0 + x - q: index x + 1 - q of the N + 1
                const unsigned pw = q ? Byte(l.w[dj - 1], x) : (x < N - 1 ? Byte(l.w[dj - 1], x + 1) : l.wN[dj - 1]);
                X[x] += (T)(pw & 0x3Fu) * R[x + 1 - q];
            }
        }
    }
#pragma unroll
    for (int x = 0; x < N; x++) X[x] *= (T)(1.0 / 64.0);
}

template <typename T, bool kX>
__device__ __forceinline__ void SplitRestrictQ(const LevelView &fv, const LevelView &cv,
                                               const uint8_t *__restrict__ pext, const T *__restrict__ res,
                                               T *__restrict__ rc, const Blk &blk)
{
    constexpr int N = kQ<T>;
    const int nq = (cv.Nz - 2 + N - 1) / N, nt = (cv.Nx - 2) * nq;
    const int t = blk.x * kPairThreads + threadIdx.x;
    if (t >= nt) return;
    const int J = 1 + t / nq, K0 = 1 + N * (t - (J - 1) * nq);
    const int S = (cv.Ny - 2 + blk.gy - 1) / blk.gy;
    const int I0 = 1 + blk.y * S, I1 = min(I0 + S, cv.Ny - 1);
    if (I0 >= I1) return;
    // a block none of whose coarse cells' children is an unknown has no coarse unknown either
    {
        const int t0 = blk.x * kPairThreads, Ja = 1 + t0 / nq, Jb = 1 + (min(t0 + kPairThreads, nt) - 1) / nq;
        const int f0 = kX ? (fv.xr[Ja] & 0x7FFF) : 2 * Ja - 1, f1 = kX ? (fv.xr[Jb] & 0x7FFF) + 1 : 2 * Jb;
        if (RowsIdle<N * kPairThreads>(fv, f0, min(f1, fv.Nx - 1), 2 * I0 - 1, min(2 * I1 - 1, fv.Ny))) return;
    }
    const bool more = K0 + N - 1 <= cv.Nz - 2; // element K0+N-1 is read only for coarse cell K0+N-1
    const RowTaps<T, kX> taps = TapsOf<T, kX>(fv, J);
    T Tm2[N], Tm1[N], Xm1[N], Xd[N];
    {
        const RestrictLoads<T> l0 = LoadRestrict<T, kX>(fv, pext, res, 2 * I0 - 2, taps, K0, more);
        const RestrictLoads<T> l1 = LoadRestrict<T, kX>(fv, pext, res, 2 * I0 - 1, taps, K0, more);
        SplitRestrictPlane<T, kX>(l0, 2 * I0 - 2, taps, Tm2, Xd);
        SplitRestrictPlane<T, kX>(l1, 2 * I0 - 1, taps, Tm1, Xm1);
    }
    for (int I = I0; I < I1; I++)
    {
        T T0[N], X0[N], T1[N], X1[N];
        const RestrictLoads<T> l0 = LoadRestrict<T, kX>(fv, pext, res, 2 * I, taps, K0, more);
        const RestrictLoads<T> l1 = LoadRestrict<T, kX>(fv, pext, res, 2 * I + 1, taps, K0, more);
        SplitRestrictPlane<T, kX>(l0, 2 * I, taps, T0, X0);
        SplitRestrictPlane<T, kX>(l1, 2 * I + 1, taps, T1, X1);
        const long long c = (long long)I * cv.sI + (long long)J * cv.sJ + K0;
#pragma unroll
        for (int x = 0; x < N; x++)
        {
            if (K0 + x <= cv.Nz - 2 && (cv.code[c + x] & CODE_UNKNOWN))
                rc[VecIdx(cv, I, J, K0 + x)] =
                    (((T)0.25 * Tm2[x] + (T)0.75 * Tm1[x]) + ((T)0.75 * T0[x] + (T)0.25 * T1[x])) + (Xm1[x] + X0[x]);
            Tm2[x] = T0[x];
            Tm1[x] = T1[x];
            Xm1[x] = X1[x];
        }
    }
}

template <typename T, bool kX>
__global__ void __launch_bounds__(kPairThreads) k_split_restrict(LevelView fv, LevelView cv,
                                                                 const uint8_t *__restrict__ pext,
                                                                 const T *__restrict__ res, T *__restrict__ rc)
{
    PdlWait();
    PdlTrigger();
    SplitRestrictQ<T, kX>(fv, cv, pext, res, rc, ThisBlk());
}

// The same restriction with one thread per coarse cell (K along the 32 lanes, J across the 8 warps), for the smaller
// coarse levels: more threads, and their launches are latency-bound.
template <typename T> struct RestrictLoads1
{
    T lo[4], hi[4];
    unsigned w[2];
};
template <typename T, bool kX>
__device__ __forceinline__ RestrictLoads1<T> LoadRestrict1(const LevelView &fv, const uint8_t *__restrict__ pext,
                                                           const T *__restrict__ res, int a, const RowTaps<T, kX> &J,
                                                           int K)
{
    RestrictLoads1<T> l;
#pragma unroll
    for (int dj = 0; dj < 4; dj++)
    {
        const long long row = (long long)min(a, fv.Ny - 1) * fv.sPS + (long long)min(J.b[dj], fv.Nx - 1) * fv.sRS + K;
        l.lo[dj] = res[row - 1];
        l.hi[dj] = res[row];
        if (dj == 1 || dj == 2) l.w[dj - 1] = pext[row - ((a + J.b[dj]) & 1)];
    }
    return l;
}

template <typename T, bool kX>
__device__ __forceinline__ void SplitRestrictPlane1(const RestrictLoads1<T> &l, int a, const RowTaps<T, kX> &J, T &Tw,
                                                   T &X)
{
    Tw = (T)0;
    X = (T)0;
#pragma unroll
    for (int dj = 0; dj < 4; dj++)
    {
        const int q = (a + J.b[dj]) & 1;
        const bool none = kX && J.w[dj] == (T)0;
        const T lo = none ? (T)0 : l.lo[dj], hi = none ? (T)0 : l.hi[dj];
        Tw += J.w[dj] * (q ? (T)0.75 * lo + (T)0.25 * hi : (T)0.25 * lo + (T)0.75 * hi);
        if (dj == 1 || (dj == 2 && J.two)) X += (T)(l.w[dj - 1] & 0x3Fu) * (q ? lo : hi);
    }
    X *= (T)(1.0 / 64.0);
}

// bx, by: the K and J tiles; bz of gz: the chunk of coarse planes
template <typename T, bool kX>
__device__ __forceinline__ void SplitRestrict1(const LevelView &fv, const LevelView &cv,
                                               const uint8_t *__restrict__ pext, const T *__restrict__ res,
                                               T *__restrict__ rc, int bx, int by, int bz, int gz)
{
    const int K = 1 + bx * 32 + threadIdx.x, J = 1 + by * 8 + threadIdx.y;
    if (K > cv.Nz - 2 || J > cv.Nx - 2) return;
    const int S = (cv.Ny - 2 + gz - 1) / gz;
    const int I0 = 1 + bz * S, I1 = min(I0 + S, cv.Ny - 1);
    if (I0 >= I1) return;
    {
        const int Ja = 1 + by * 8, Jb = min(Ja + 7, cv.Nx - 2); // idle as SplitRestrictQ's
        const int f0 = kX ? (fv.xr[Ja] & 0x7FFF) : 2 * Ja - 1, f1 = kX ? (fv.xr[Jb] & 0x7FFF) + 1 : 2 * Jb;
        if (RowsIdle<kQ<T> * kPairThreads>(fv, f0, min(f1, fv.Nx - 1), 2 * I0 - 1, min(2 * I1 - 1, fv.Ny))) return;
    }
    const RowTaps<T, kX> taps = TapsOf<T, kX>(fv, J);
    T Tm2, Tm1, Xm1, Xdummy;
    {
        const RestrictLoads1<T> l0 = LoadRestrict1<T, kX>(fv, pext, res, 2 * I0 - 2, taps, K);
        const RestrictLoads1<T> l1 = LoadRestrict1<T, kX>(fv, pext, res, 2 * I0 - 1, taps, K);
        SplitRestrictPlane1<T, kX>(l0, 2 * I0 - 2, taps, Tm2, Xdummy);
        SplitRestrictPlane1<T, kX>(l1, 2 * I0 - 1, taps, Tm1, Xm1);
    }
    for (int I = I0; I < I1; I++)
    {
        T T0, X0, T1, X1;
        const RestrictLoads1<T> l0 = LoadRestrict1<T, kX>(fv, pext, res, 2 * I, taps, K);
        const RestrictLoads1<T> l1 = LoadRestrict1<T, kX>(fv, pext, res, 2 * I + 1, taps, K);
        SplitRestrictPlane1<T, kX>(l0, 2 * I, taps, T0, X0);
        SplitRestrictPlane1<T, kX>(l1, 2 * I + 1, taps, T1, X1);
        const long long c = (long long)I * cv.sI + (long long)J * cv.sJ + K;
        if (cv.code[c] & CODE_UNKNOWN)
            rc[VecIdx(cv, I, J, K)] = (((T)0.25 * Tm2 + (T)0.75 * Tm1) + ((T)0.75 * T0 + (T)0.25 * T1)) + (Xm1 + X0);
        Tm2 = T0;
        Tm1 = T1;
        Xm1 = X1;
    }
}

template <typename T, bool kX>
__global__ void __launch_bounds__(256) k_split_restrict1(LevelView fv, LevelView cv, const uint8_t *__restrict__ pext,
                                                        const T *__restrict__ res, T *__restrict__ rc)
{
    PdlWait();
    PdlTrigger();
    SplitRestrict1<T, kX>(fv, cv, pext, res, rc, (int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, (int)gridDim.z);
}

// Coarse levels with at least kRestrictQuadCells cells take the quad kernel (4x fewer loads per coarse cell), the
// smaller ones the per-cell kernel (mode 0); mode 1 takes the per-cell kernel and mode 2 the quad kernel everywhere.
// Both sum the same products in the same order. Restriction from 194^3, 162^3, 130^3 and 98^3, per cell against quads
// (B200, us): FP32 17.9 / 15.6, 15.8 / 13.4, 11.6 / 9.8, 9.6 / 9.4; FP64 25.1 / 17.8, 16.5 / 15.3, 15.5 / 12.2,
// 9.5 / 9.6. The line lies between the last two (coarse levels of 66^3 and 50^3).
constexpr long long kRestrictQuadCells = 1LL << 17;

template <typename T, bool kX>
static void RestrictOn(const LevelView &fine, const LevelView &coarse, const uint8_t *pext, const T *resFine,
                       T *rCoarse, int mode, cudaStream_t st)
{
    if (mode == 1 || (mode != 2 && coarse.cells < kRestrictQuadCells))
    {
        const long long perPlane = (long long)((coarse.Nz - 2 + 31) / 32) * ((coarse.Nx - 2 + 7) / 8);
        const int S = MarchPlanes(coarse.Ny - 2, perPlane);
        const dim3 grid((unsigned)((coarse.Nz - 2 + 31) / 32), (unsigned)((coarse.Nx - 2 + 7) / 8),
                        (unsigned)((coarse.Ny - 2 + S - 1) / S));
        LaunchPdl(k_split_restrict1<T, kX>, grid, dim3(32, 8), 0, st, fine, coarse, pext, resFine, rCoarse);
        return;
    }
    const long long nt = (long long)(coarse.Nx - 2) * ((coarse.Nz - 2 + kQ<T> - 1) / kQ<T>);
    const long long perPlane = (nt + kPairThreads - 1) / kPairThreads, planes = coarse.Ny - 2 > 0 ? coarse.Ny - 2 : 1;
    const long long bestS = BestMarch(perPlane, planes, (long long)SmCount() * Occ<k_split_restrict<T, kX>>());
    LaunchPdl(k_split_restrict<T, kX>, dim3((unsigned)perPlane, (unsigned)((planes + bestS - 1) / bestS)),
              kPairThreads, 0, st, fine, coarse, pext, resFine, rCoarse);
}

template <typename T>
void LaunchSplitRestrict(const LevelView &fine, const LevelView &coarse, const uint8_t *pext, const T *resFine,
                         T *rCoarse, int mode, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if constexpr (sizeof(T) == 8) // stretched grids run on this layout in FP64
        if (fine.xr) return RestrictOn<T, true>(fine, coarse, pext, resFine, rCoarse, mode, st);
    RestrictOn<T, false>(fine, coarse, pext, resFine, rCoarse, mode, st);
}

// ---------------------------------------------------------------------------------------------------------------
// PCG on a split level 0 (the semantics of k_pair_papply)
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ double SplitRzEff(const double *S, int base, double n, int singular)
{
    return singular ? S[base] - (S[base + 1] / n) * S[base + 2] : S[base];
}

// p_new = U (z - mean + beta p_old), q = M p_new, sum p_new.q, both colours at a thread's quad position.
template <typename T, bool kSingular>
__device__ __forceinline__ void SplitPApply(const LevelView &v, const uint8_t *__restrict__ du,
                                            const T *__restrict__ z, T *p0, T *p1, T *__restrict__ q,
                                            const Reducer &R, const double *S, const int *it, int baseEven,
                                            int baseOdd, int slotN, int slotPQ, const Blk &blk)
{
    constexpr int N = kQ<T>;
    const int iter = *it, par = iter & 1;
    const T *__restrict__ pIn = par ? p1 : p0;
    T *__restrict__ pOut = par ? p0 : p1;
    const int baseNew = par ? baseOdd : baseEven, baseOld = par ? baseEven : baseOdd;
    const double n = S[slotN];
    const double beta =
        iter == 0 ? 0.0 : SplitRzEff(S, baseNew, n, kSingular) / SplitRzEff(S, baseOld, n, kSingular);
    const T bt = (T)beta;
    const T mean = kSingular ? (T)(S[baseNew + 1] / n) : (T)0;
    const QuadPos P = QuadStart<N>(v, blk);
    if (TileIdle(v, blk.x, P.i0, P.i1))
    {
        double zero[1] = {0.0}; // p and q stay zero on these cells; the block adds its zero term to p.q
        GridReduceB<1>(R, zero, slotPQ, BlkId(blk), BlkCount(blk));
        return;
    }
    const T g = (T)v.gamma, hg = (T)0.5 * (T)v.gamma;
    const long long hb = v.sHalf;
    auto pn = [&](long long base) {
        const Quad<T> zz = LQ(z + base), pv = LQ(pIn + base);
        Quad<T> out;
#pragma unroll
        for (int x = 0; x < N; x++) out.v[x] = (zz.v[x] - mean) + bt * pv.v[x];
        if (kSingular)
        {
            const unsigned d = LdB<N>(du + base);
#pragma unroll
            for (int x = 0; x < N; x++) out.v[x] *= Unk<T>(Byte(d, x));
        }
        return out;
    };
    auto pn1 = [&](long long idx) {
        T x = (z[idx] - mean) + bt * pIn[idx];
        if (kSingular) x *= Unk<T>(du[idx]);
        return x;
    };
    const long long b0 = P.off, b1 = hb + P.off;
    Quad<T> M0 = pn(b0 - P.PS), M1 = pn(b1 - P.PS), C0 = pn(b0), C1 = pn(b1);
    T facc = (T)0;
    long long o = 0;
    for (int i = P.i0; i < P.i1; i++, o += P.PS)
    {
        const Quad<T> P0 = pn(b0 + o + P.PS), P1 = pn(b1 + o + P.PS);
        const Quad<T> Jp0 = pn(b0 + o + P.RS), Jp1 = pn(b1 + o + P.RS), Jm0 = pn(b0 + o - P.RS), Jm1 = pn(b1 + o - P.RS);
        const unsigned d0 = LdB<N>(du + b0 + o), d1 = LdB<N>(du + b1 + o);
        const int q0 = (i + P.j) & 1, q1 = q0 ^ 1;
        T pw0 = __shfl_up_sync(0xffffffffu, C0.v[N - 1], 1), nx0 = __shfl_down_sync(0xffffffffu, C0.v[0], 1);
        T pw1 = __shfl_up_sync(0xffffffffu, C1.v[N - 1], 1), nx1 = __shfl_down_sync(0xffffffffu, C1.v[0], 1);
        if (P.lane == 0 && P.m0 > 0)
        {
            pw0 = pn1(b0 + o - 1);
            pw1 = pn1(b1 + o - 1);
        }
        if (P.lane == 31 && P.m0 + N < P.RS)
        {
            nx0 = pn1(b0 + o + N);
            nx1 = pn1(b1 + o + N);
        }
        // colour-0 cells see colour 1 shifted by q0, colour-1 cells see colour 0 shifted by q1
        const Quad<T> sh1 = KShift(C1, pw1, nx1, q0), sh0 = KShift(C0, pw0, nx0, q1);
        Quad<T> Q0, Q1;
#pragma unroll
        for (int x = 0; x < N; x++)
        {
            const unsigned a0 = Byte(d0, x), a1 = Byte(d1, x);
            const T s0 = ((P1.v[x] + M1.v[x]) + (Jp1.v[x] + Jm1.v[x])) + (C1.v[x] + sh1.v[x]);
            const T s1 = ((P0.v[x] + M0.v[x]) + (Jp0.v[x] + Jm0.v[x])) + (C0.v[x] + sh0.v[x]);
            Q0.v[x] = Unk<T>(a0) * (hg * (T)(a0 & 0x7Fu) * C0.v[x] - g * s0);
            Q1.v[x] = Unk<T>(a1) * (hg * (T)(a1 & 0x7Fu) * C1.v[x] - g * s1);
        }
        if (P.valid)
        {
            SQ(pOut + b0 + o, C0);
            SQ(pOut + b1 + o, C1);
            SQ(q + b0 + o, Q0);
            SQ(q + b1 + o, Q1);
#pragma unroll
            for (int x = 0; x < N; x++) facc += C0.v[x] * Q0.v[x] + C1.v[x] * Q1.v[x];
        }
        M0 = C0;
        M1 = C1;
        C0 = P0;
        C1 = P1;
    }
    double acc[1] = {facc};
    GridReduceB<1>(R, acc, slotPQ, BlkId(blk), BlkCount(blk));
}

// FP64: 3 resident blocks (64 registers spill 132 bytes)
template <typename T, bool kSingular>
__global__ void __launch_bounds__(kPairThreads, sizeof(T) == 8 ? 3 : 4)
    k_split_papply(LevelView v, const uint8_t *__restrict__ du, const T *__restrict__ z, T *p0, T *p1,
                   T *__restrict__ q, Reducer R, const double *S, const int *it, int baseEven, int baseOdd,
                   int slotN, int slotPQ)
{
    PdlWait();
    PdlTrigger();
    SplitPApply<T, kSingular>(v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, slotPQ, ThisBlk());
}

template <typename T>
void LaunchSplitPApply(const LevelView &v, const uint8_t *du, const T *z, T *p0, T *p1, T *q,
                       const Reducer &R, const double *S, const int *it, int baseEven, int baseOdd, int slotN,
                       int singular, int slotPQ, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8)
        if (v.stretched)
            return LaunchStretchedPApply(v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, singular, slotPQ, st);
    NB_COUNT_LAUNCH();
    if (singular)
        LaunchPdl(k_split_papply<T, true>, SumGrid(R, QuadGrid<kQ<T>>(v, Occ<k_split_papply<T, true>>())), kPairThreads, 0,
                  st, v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, slotPQ);
    else
        LaunchPdl(k_split_papply<T, false>, SumGrid(R, QuadGrid<kQ<T>>(v, Occ<k_split_papply<T, false>>())), kPairThreads,
                  0, st, v, du, z, p0, p1, q, R, S, it, baseEven, baseOdd, slotN, slotPQ);
}

// ---------------------------------------------------------------------------------------------------------------
// the outer FP64 side of level 0: FP64 arrays in the grid layout, the solver's vectors (T) colour-split
// ---------------------------------------------------------------------------------------------------------------
// The two cells (i, j, k0), (i, j, k0 + 1), k0 even, of an FP64 grid-layout array: one aligned 16-byte access with Nz
// even; with Nz odd two 8-byte ones, the second left out (and read as zero) past the row's last cell (two = false).
template <bool kEven> __device__ __forceinline__ double2 LdPair(const double *p, bool two)
{
    if constexpr (kEven) return *reinterpret_cast<const double2 *>(p);
    else return make_double2(p[0], two ? p[1] : 0.0);
}
template <bool kEven> __device__ __forceinline__ void StPair64(double *p, const double2 &x, bool two)
{
    if constexpr (kEven) *reinterpret_cast<double2 *>(p) = x;
    else
    {
        p[0] = x.x;
        if (two) p[1] = x.y;
    }
}

// r = sfac * b (split) and (sum b^2, sum b): the residual of a zero iterate. One thread per cell pair (k0 even).
// bx of gx: this block among the launch's blocks (a grid-stride loop)
template <typename T, bool kEven>
__device__ __forceinline__ void SplitScaleSum(const LevelView &v, const double *__restrict__ b, T *__restrict__ r,
                                              double sfac, const Reducer &R, int slot, int bx, int gx)
{
    double acc[2] = {0.0, 0.0};
    const int H = (v.Nz + 1) >> 1;
    const long long pairs = (long long)v.Ny * v.Nx * H, stride = (long long)gx * blockDim.x;
    for (long long t = bx * (long long)blockDim.x + threadIdx.x; t < pairs; t += stride)
    {
        const long long row = t / H; // i * Nx + j
        const int m = (int)(t - row * H);
        const double2 x = LdPair<kEven>(b + row * v.Nz + 2 * m, 2 * m + 1 < v.Nz);
        const int i = (int)(row / v.Nx), j = (int)(row - (long long)i * v.Nx);
        const int par = (i + j) & 1; // the colour of the pair's first cell
        const long long s = (long long)i * v.sPS + (long long)j * v.sRS + m;
        r[par * v.sHalf + s] = (T)(x.x * sfac);
        r[(par ^ 1) * v.sHalf + s] = (T)(x.y * sfac);
        acc[0] += x.x * x.x + x.y * x.y;
        acc[1] += x.x + x.y;
    }
    GridReduceB<2>(R, acc, slot, (unsigned)bx, (unsigned)gx);
}

constexpr int kScaleSumBlocks = 148 * 8;

template <typename T, bool kEven>
__global__ void __launch_bounds__(256) k_split_scale_sum(LevelView v, const double *__restrict__ b,
                                                         T *__restrict__ r, double sfac, Reducer R, int slot)
{
    SplitScaleSum<T, kEven>(v, b, r, sfac, R, slot, (int)blockIdx.x, (int)gridDim.x);
}

template <typename T>
void LaunchSplitScaleSum(const LevelView &v, const double *b, T *r, double sfac, const Reducer &R, int slot,
                         cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if (v.Nz % 2 == 0) k_split_scale_sum<T, true><<<kScaleSumBlocks, 256, 0, st>>>(v, b, r, sfac, R, slot);
    else k_split_scale_sum<T, false><<<kScaleSumBlocks, 256, 0, st>>>(v, b, r, sfac, R, slot);
}

// The FP64 refinement step on a uniform split level 0 (k_pair_refine64's, with e read and r written split):
// x_out = x_in + e; r = sfac (b - A x_out) in T; (sum (b - A x_out)^2, sum (b - A x_out)) in FP64. One thread per
// cell pair of the grid layout; the pair (k0, k0+1) of row (i, j) is element k0/2 of colours (i+j)&1 and its other.
// cell pairs of a row, and the position of a thread's pair with Nz odd (PairStart's with Nz even)
__device__ __host__ __forceinline__ int RowPairs(const LevelView &v) { return (v.Nz + 1) >> 1; }

template <bool kEven> __device__ __forceinline__ PairPos RowPairStart(const LevelView &v, const Blk &b)
{
    PairPos p = PairStart(v, b.x, b.y, b.gy);
    if constexpr (!kEven)
    {
        const int H = RowPairs(v), P = v.Nx * H;
        int q = b.x * kPairThreads + threadIdx.x;
        p.valid = q < P;
        if (!p.valid) q = P - 1;
        p.j = q / H;
        p.k0 = 2 * (q - p.j * H);
        p.base = (long long)p.i0 * v.sI + (long long)p.j * v.sJ + p.k0;
    }
    return p;
}

// 3 resident blocks (80 registers, no spill) beat 4 with a 64-register cap that spills (measured 115 vs 122 us)
template <typename T, bool kEven>
__device__ __forceinline__ void SplitRefine64(const LevelView &v, const uint8_t *__restrict__ du,
                                              const double *__restrict__ b, const double *__restrict__ xin,
                                              const T *__restrict__ e, double *__restrict__ xout,
                                              T *__restrict__ r, double scale, double sfac, const Reducer &R,
                                              int slot, const Blk &blk)
{
    const PairPos P = RowPairStart<kEven>(v, blk);
    const bool in2 = kEven || P.k0 + 1 < v.Nz; // the pair has a second cell
    if (v.act)
    {
        // the block's pairs lie in rows j0 .. j1; with no unknown there, x_out = x_in + e and r stay zero
        const int q0 = kPairThreads * blk.x, H = RowPairs(v);
        const int j0 = q0 / H, j1 = min(v.Nx - 1, (q0 + kPairThreads - 1) / H);
        if (RowsIdle<kQ<T> * kPairThreads>(v, j0, j1, P.i0, P.i1))
        {
            double zero[2] = {0.0, 0.0};
            GridReduceB<2>(R, zero, slot, BlkId(blk), BlkCount(blk));
            return;
        }
    }
    const long long sb = (long long)P.i0 * v.sPS + (long long)P.j * v.sRS + (P.k0 >> 1);
    // the thread's element on plane i0 in colour 0 and colour 1
    const T *e0 = e + sb, *e1 = e + v.sHalf + sb;
    const uint8_t *d0p = du + sb, *d1p = du + v.sHalf + sb;
    T *r0p = r + sb, *r1p = r + v.sHalf + sb;
    const double *xp = xin + P.base;
    // x_in + e at the pair `o` cells (grid layout) / `so` elements (split) away; par: the colour of its first cell
    auto X = [&](long long o, long long so, int par) {
        const double2 a = LdPair<kEven>(xp + o, in2);
        const T fa = e0[so], fb = e1[so];
        return make_double2(a.x + (double)(par ? fb : fa), a.y + (double)(par ? fa : fb));
    };
    const int par0 = (P.i0 + P.j) & 1;
    double2 XM = X(-P.sI, -v.sPS, par0 ^ 1), XC = X(0, 0, par0);
    double acc[2] = {0.0, 0.0};
    long long off = 0, so = 0;
    for (int i = P.i0; i < P.i1; i++, off += P.sI, so += v.sPS)
    {
        const int par = (i + P.j) & 1;
        const double2 XP = X(off + P.sI, so + v.sPS, par ^ 1);
        const double2 XJp = X(off + P.sJ, so + v.sRS, par ^ 1), XJm = X(off - P.sJ, so - v.sRS, par ^ 1);
        const double2 bb = LdPair<kEven>(b + P.base + off, in2);
        const unsigned da = d0p[so], db = d1p[so];
        const unsigned d0 = par ? db : da, d1 = par ? da : db;
        double left = __shfl_up_sync(0xffffffffu, XC.y, 1);
        double right = __shfl_down_sync(0xffffffffu, XC.x, 1);
        // cell k0-1 is element m-1 of the other colour, cell k0+2 element m+1 of this one (across a row's end: a ring
        // cell's neighbour, masked)
        if (P.lane == 0) left = xp[off - 1] + (double)(par ? e0[so - 1] : e1[so - 1]);
        if (P.lane == 31) right = xp[off + 2] + (double)(par ? e1[so + 1] : e0[so + 1]);
        const double s0 = ((XP.x + XM.x) + (XJp.x + XJm.x)) + (left + XC.y);
        const double s1 = ((XP.y + XM.y) + (XJp.y + XJm.y)) + (XC.x + right);
        const double r0 = (d0 & 0x80u) ? bb.x - scale * (s0 - 0.5 * (double)(d0 & 0x7Fu) * XC.x) : 0.0;
        const double r1 = (d1 & 0x80u) ? bb.y - scale * (s1 - 0.5 * (double)(d1 & 0x7Fu) * XC.y) : 0.0;
        if (P.valid)
        {
            StPair64<kEven>(xout + P.base + off, XC, in2);
            const T f0 = (T)(r0 * sfac), f1 = (T)(r1 * sfac);
            r0p[so] = par ? f1 : f0;
            r1p[so] = par ? f0 : f1;
            acc[0] += r0 * r0 + r1 * r1;
            acc[1] += r0 + r1;
        }
        XM = XC;
        XC = XP;
    }
    GridReduceB<2>(R, acc, slot, BlkId(blk), BlkCount(blk));
}

// swap (may be null): when *swap is odd, x_in and x_out trade places
template <typename T, bool kEven>
__global__ void __launch_bounds__(kPairThreads, 3)
    k_split_refine64(LevelView v, const uint8_t *__restrict__ du, const double *__restrict__ b,
                     const double *xin, const T *__restrict__ e, double *xout,
                     T *__restrict__ r, double scale, double sfac, Reducer R, int slot, const int *swap)
{
    const bool sw = swap && (*swap & 1);
    SplitRefine64<T, kEven>(v, du, b, sw ? xout : xin, e, sw ? const_cast<double *>(xin) : xout, r, scale, sfac, R, slot,
                  ThisBlk());
}

template <typename T>
void LaunchSplitRefine64(const LevelView &v, const uint8_t *du, const double *b, const double *xin, const T *e,
                         double *xout, T *r, double scale, double sfac, const Reducer &R, int slot,
                         cudaStream_t st, const int *swap)
{
    NB_COUNT_LAUNCH();
    const dim3 grid = SumGrid(R, PairGridOf((long long)v.Nx * RowPairs(v), v.Ny - 2, kSumPlanes));
    if (v.Nz % 2 == 0)
        k_split_refine64<T, true><<<grid, kPairThreads, 0, st>>>(v, du, b, xin, e, xout, r, scale, sfac, R, slot, swap);
    else
        k_split_refine64<T, false><<<grid, kPairThreads, 0, st>>>(v, du, b, xin, e, xout, r, scale, sfac, R, slot,
                                                                  swap);
}

// The most blocks such a launch takes: a quad kernel with two doubles a thread, on kQuadMaxS planes where that fills ten
// waves (BestMarch stops there; with fewer waves, the longest shorter march has at most twice the blocks of one that fills
// less than ten), or a pair-thread one.
long long SplitSumBlocks(const LevelView &v)
{
    const long long few = 2LL * 10 * 148 * 8;
    const dim3 q = QuadGridS<2>(v, kQuadMaxS), p = PairGridOf((long long)v.Nx * RowPairs(v), v.Ny - 2, kSumPlanes);
    return std::max(few, std::max((long long)q.x * q.y, (long long)p.x * p.y));
}

// ---------------------------------------------------------------------------------------------------------------
// batched launches (nb_batch.cu): grid z = the batch's capacity, block z runs the request at list[z] on the x, y tiles
// of its own grid. The launches that end in a grid-wide sum keep the grid a single solve uses, so each request's sums
// run over its own blocks in the same order whatever else the batch holds; the others take the march length S the
// caller chose (it changes which planes a thread visits, not what a cell gets).
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kPairThreads, 4) kb_split_first(const BatchLevel *__restrict__ lv, int ls, int l,
                                                               BatchList a)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls + l];
    SplitFirst<float>(L.v, L.du, L.r, L.e, ThisBlk());
}

template <int kDot>
__global__ void __launch_bounds__(kPairThreads, kDot ? 3 : 4)
    kb_split_half(const BatchLevel *__restrict__ lv, int ls, int l, const BatchReq *__restrict__ rq, BatchList a,
                  int colour, int baseEven, int baseOdd, int partSlot)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls + l];
    const long long h = L.v.sHalf;
    if (kDot)
        SplitHalf<float, kDot>(L.v, L.du + colour * h, L.r + colour * h, L.e + (colour ^ 1) * h, L.e + colour * h, colour,
                        rq[q].red, rq[q].it, baseEven, baseOdd, partSlot, ThisBlk());
    else
        SplitHalf<float, kDot>(L.v, L.du + colour * h, L.r + colour * h, L.e + (colour ^ 1) * h, L.e + colour * h, colour,
                        Reducer{}, nullptr, baseEven, baseOdd, partSlot, ThisBlk());
}

__global__ void __launch_bounds__(kPairThreads, 3) kb_split_residual(const BatchLevel *__restrict__ lv, int ls, int l,
                                                                  BatchList a)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls + l];
    SplitResidual<float>(L.v, L.du, L.r, L.e, L.res, ThisBlk());
}

__global__ void __launch_bounds__(kPairThreads) kb_split_prolong(const BatchLevel *__restrict__ lv, int ls, int l,
                                                                 BatchList a)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &F = lv[q * ls + l], &C = lv[q * ls + l + 1];
    SplitProlong<float, false>(F.v, C.v, F.pext, C.e, F.e, ThisBlk());
}

__global__ void __launch_bounds__(kPairThreads) kb_split_restrict(const BatchLevel *__restrict__ lv, int ls, int l,
                                                                  BatchList a)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &F = lv[q * ls + l], &C = lv[q * ls + l + 1];
    SplitRestrictQ<float, false>(F.v, C.v, F.pext, F.res, C.r, ThisBlk());
}

// grid (K tiles, J tiles x gz plane chunks, capacity)
__global__ void __launch_bounds__(256) kb_split_restrict1(const BatchLevel *__restrict__ lv, int ls, int l,
                                                         BatchList a, int gyJ, int gz)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &F = lv[q * ls + l], &C = lv[q * ls + l + 1];
    const int by = (int)blockIdx.y % gyJ, bz = (int)blockIdx.y / gyJ;
    SplitRestrict1<float, false>(F.v, C.v, F.pext, F.res, C.r, (int)blockIdx.x, by, bz, gz);
}

// The requests of one form (singular or not), each form in a kernel and a launch of its own: both inlined into one
// kernel took 64 registers with 552 bytes spilled, apart they spill 128 and 180 at 80 registers. 16 tanks of 128^3, the
// step: 16.1 ms in one kernel, 15.8 apart at 3 blocks an SM, 16.2 at 2.
template <bool kSingular>
__global__ void __launch_bounds__(kPairThreads, 3)
    kb_split_papply(const BatchLevel *__restrict__ lv, int ls, const BatchReq *__restrict__ rq, BatchList a,
                    int baseEven, int baseOdd, int slotN, int slotPQ)
{
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls];
    const BatchReq &Q = rq[q];
    if ((Q.singular != 0) != kSingular) return;
    SplitPApply<float, kSingular>(L.v, L.du, L.e, Q.p0, Q.p1, Q.q, Q.red, Q.red.out, Q.it, baseEven, baseOdd, slotN,
                                  slotPQ, ThisBlk());
}

__global__ void __launch_bounds__(256) kb_split_scale_sum(const BatchLevel *__restrict__ lv, int ls,
                                                          const BatchReq *__restrict__ rq, BatchList a, int slot)
{
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls];
    const BatchReq &Q = rq[q];
    SplitScaleSum<float, true>(L.v, Q.b, L.r, Q.sfac, Q.red, slot, (int)blockIdx.x, (int)gridDim.x);
}

// parity[q]: this pass reads x from xin (0) or xout (1) and writes the other
__global__ void __launch_bounds__(kPairThreads, 3)
    kb_split_refine64(const BatchLevel *__restrict__ lv, int ls, const BatchReq *__restrict__ rq, BatchList a,
                      const int *__restrict__ parity, int slot)
{
    const int q = BatchReqOf(a);
    if (q < 0) return;
    const BatchLevel &L = lv[q * ls];
    const BatchReq &Q = rq[q];
    const bool odd = parity[q] & 1;
    SplitRefine64<float, true>(L.v, L.du, Q.b, odd ? Q.xout : Q.xin, Q.x, odd ? Q.xin : Q.xout, L.r, Q.scale, Q.sfac,
                               Q.red, slot, ThisBlk());
}

namespace
{
inline dim3 WithZ(dim3 g, int cap)
{
    g.z = (unsigned)cap;
    return g;
}
} // namespace

// the march length a quad kernel's single launch takes on this colour-split level (the default of the batched
// smoothing and residual launches)
int SplitDefaultS(const LevelView &v, int kind)
{
    int occ = 1;
    switch (kind)
    {
    case NB_BK_FIRST: occ = Occ<k_split_first<float>>(); break;
    case NB_BK_HALF: occ = Occ<k_split_half<float, 0>>(); break;
    default: occ = Occ<k_split_residual<float>>(); break;
    }
    const long long planes = v.Ny - 2 > 0 ? v.Ny - 2 : 1;
    const dim3 g = QuadGrid<4>(v, occ);
    return (int)((planes + g.y - 1) / g.y);
}

void LaunchBatchSplit(int kind, const LevelView &v, const LevelView *coarse, int S, int mode,
                      const BatchLevel *lv, int ls, int l, const BatchReq *rq, BatchList a, int cap, int colour,
                      cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    S = S < 1 ? 1 : S;
    switch (kind)
    {
    case NB_BK_FIRST:
        LaunchPdl(kb_split_first, WithZ(QuadGridS<4>(v, S), cap), kPairThreads, 0, st, lv, ls, l, a);
        break;
    case NB_BK_HALF:
        LaunchPdl(kb_split_half<0>, WithZ(QuadGridS<4>(v, S), cap), kPairThreads, 0, st, lv, ls, l, rq, a, colour, 0, 0,
                  0);
        break;
    case NB_BK_RESIDUAL:
        LaunchPdl(kb_split_residual, WithZ(QuadGridS<4>(v, S), cap), kPairThreads, 0, st, lv, ls, l, a);
        break;
    case NB_BK_PROLONG:
        LaunchPdl(kb_split_prolong, WithZ(ProlongGridS<4>(v, *coarse, S), cap), kPairThreads, 0, st, lv, ls, l, a);
        break;
    case NB_BK_RESTRICT:
    {
        const LevelView &c = *coarse;
        const long long planes = c.Ny - 2 > 0 ? c.Ny - 2 : 1;
        const int gz = (int)((planes + S - 1) / S);
        if (mode == 1)
        {
            const int gx = (c.Nz - 2 + 31) / 32, gyJ = (c.Nx - 2 + 7) / 8;
            LaunchPdl(kb_split_restrict1, dim3((unsigned)gx, (unsigned)(gyJ * gz), (unsigned)cap), dim3(32, 8), 0,
                      st, lv, ls, l, a, gyJ, gz);
        }
        else
        {
            const long long nt = (long long)(c.Nx - 2) * ((c.Nz - 2 + 3) / 4);
            const long long perPlane = (nt + kPairThreads - 1) / kPairThreads;
            LaunchPdl(kb_split_restrict, dim3((unsigned)perPlane, (unsigned)gz, (unsigned)cap), kPairThreads, 0, st,
                      lv, ls, l, a);
        }
        break;
    }
    default: break;
    }
}

// The launches that end in a grid-wide sum, on the grids a single solve of the level uses.
void LaunchBatchSplitHalfDot(const LevelView &v, const BatchLevel *lv, int ls, const BatchReq *rq, BatchList a,
                             int cap, int colour, bool last, int baseEven, int baseOdd, int partSlot, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if (last)
        LaunchPdl(kb_split_half<2>, WithZ(QuadGrid<4>(v, Occ<k_split_half<float, 2>>()), cap), kPairThreads, 0, st, lv, ls, 0,
                  rq, a, colour, baseEven, baseOdd, partSlot);
    else
        LaunchPdl(kb_split_half<1>, WithZ(QuadGrid<4>(v, Occ<k_split_half<float, 1>>()), cap), kPairThreads, 0, st, lv, ls, 0,
                  rq, a, colour, baseEven, baseOdd, partSlot);
}

// forms: bit 0, some request is not singular; bit 1, some request is. Each on the grid a single solve of its form uses.
void LaunchBatchSplitPApply(const LevelView &v, const BatchLevel *lv, int ls, const BatchReq *rq, BatchList a,
                            int cap, int baseEven, int baseOdd, int slotN, int slotPQ, int forms, cudaStream_t st)
{
    if (forms & 1)
    {
        NB_COUNT_LAUNCH();
        LaunchPdl(kb_split_papply<false>, WithZ(QuadGrid<4>(v, Occ<k_split_papply<float, false>>()), cap), kPairThreads, 0,
                  st, lv, ls, rq, a, baseEven, baseOdd, slotN, slotPQ);
    }
    if (forms & 2)
    {
        NB_COUNT_LAUNCH();
        LaunchPdl(kb_split_papply<true>, WithZ(QuadGrid<4>(v, Occ<k_split_papply<float, true>>()), cap), kPairThreads, 0,
                  st, lv, ls, rq, a, baseEven, baseOdd, slotN, slotPQ);
    }
}

void LaunchBatchSplitScaleSum(const BatchLevel *lv, int ls, const BatchReq *rq, BatchList a, int cap, int slot,
                              cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    kb_split_scale_sum<<<dim3(kScaleSumBlocks, 1, cap), 256, 0, st>>>(lv, ls, rq, a, slot);
}

void LaunchBatchSplitRefine64(const LevelView &v, const BatchLevel *lv, int ls, const BatchReq *rq, BatchList a,
                              int cap, const int *parity, int slot, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    kb_split_refine64<<<WithZ(PairGrid(v, kSumPlanes), cap), kPairThreads, 0, st>>>(lv, ls, rq, a, parity, slot);
}

// ---------------------------------------------------------------------------------------------------------------
// tile activity: one warp per (plane, tile), ORing the unknown bits of the tile's diagonal bytes in both colours. One
// thread per tile read its 2 KB word by word, a few blocks of latency per level of every layout change (130^3 and its
// three coarser split levels, B200: 290 -> 15 us).
// ---------------------------------------------------------------------------------------------------------------
static int TileElems(int elemBytes) { return 16 / elemBytes * kPairThreads; }

int SplitActivityTiles(const LevelView &v, int elemBytes)
{
    return (v.sPS + TileElems(elemBytes) - 1) / TileElems(elemBytes);
}

__global__ void __launch_bounds__(256) k_split_activity(LevelView v, const uint8_t *__restrict__ du,
                                                        uint8_t *__restrict__ act, int tiles, int tileElems)
{
    const int lane = threadIdx.x & 31;
    const long long t = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= (long long)v.Ny * tiles) return;
    const int i = (int)(t / tiles), tile = (int)(t - (long long)i * tiles);
    const int e0 = tile * tileElems, e1 = min(e0 + tileElems, v.sPS);
    const uint8_t *row0 = du + (long long)i * v.sPS, *row1 = row0 + v.sHalf;
    unsigned any = 0;
#pragma unroll 4
    for (int e = e0 + 4 * lane; e < e1; e += 128) any |= LdB<4>(row0 + e) | LdB<4>(row1 + e); // sPS, e0: multiples of 4
    any = __any_sync(0xffffffffu, (any & 0x80808080u) != 0);
    if (lane == 0) act[t] = any ? 1 : 0;
}

void LaunchSplitActivity(const LevelView &v, const uint8_t *du, uint8_t *act, int tiles, int elemBytes,
                         cudaStream_t st)
{
    const long long n = (long long)v.Ny * tiles;
    NB_COUNT_LAUNCH();
    k_split_activity<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(v, du, act, tiles, TileElems(elemBytes));
}

// The occupancy of every split kernel, read outside any stream capture (the launchers size their grids from it).
template <typename T> static void PrepareSplit()
{
    (void)Occ<k_split_first<T>>();
    (void)Occ<k_split_half<T, 0>>();
    (void)Occ<k_split_half<T, 1>>();
    (void)Occ<k_split_half<T, 2>>();
    (void)Occ<k_split_residual<T>>();
    (void)Occ<k_split_prolong<T, false>>();
    (void)Occ<k_split_restrict<T, false>>();
    (void)Occ<k_split_papply<T, true>>();
    (void)Occ<k_split_papply<T, false>>();
}

void PrepareSplitKernels(int elemBytes)
{
    if (elemBytes == 8)
    {
        PrepareSplit<double>();
        (void)Occ<k_split_prolong<double, true>>();
        (void)Occ<k_split_restrict<double, true>>();
        PrepareStretchedKernels();
    }
    else PrepareSplit<float>();
}

#define NB_INST(T)                                                                                                 \
    template void LaunchSplitFirst<T>(const LevelView &, const uint8_t *, const T *, T *, cudaStream_t);           \
    template void LaunchSplitHalf<T>(const LevelView &, const uint8_t *, const T *, T *, int, cudaStream_t);       \
    template void LaunchSplitHalfDot<T>(const LevelView &, const uint8_t *, const T *, T *, int, bool,             \
                                        const Reducer &, const int *, int, int, int, cudaStream_t);                \
    template void LaunchSplitResidual<T>(const LevelView &, const uint8_t *, const T *, const T *, T *,            \
                                         cudaStream_t);                                                            \
    template void LaunchSplitProlong<T>(const LevelView &, const LevelView &, const uint8_t *, const T *, T *,     \
                                        cudaStream_t);                                                             \
    template void LaunchSplitRestrict<T>(const LevelView &, const LevelView &, const uint8_t *, const T *, T *,    \
                                         int, cudaStream_t);                                                       \
    template void LaunchSplitPApply<T>(const LevelView &, const uint8_t *, const T *, T *, T *, T *,               \
                                       const Reducer &, const double *, const int *, int, int, int, int, int,      \
                                       cudaStream_t);                                                              \
    template void LaunchSplitScaleSum<T>(const LevelView &, const double *, T *, double, const Reducer &, int,     \
                                         cudaStream_t);                                                            \
    template void LaunchSplitRefine64<T>(const LevelView &, const uint8_t *, const double *, const double *,       \
                                         const T *, double *, T *, double, double, const Reducer &, int,           \
                                         cudaStream_t, const int *);
NB_INST(float)
NB_INST(double)
#undef NB_INST

} // namespace nb
