// The two legs of the V-cycle on a small uniform colour-split level, one kernel each: the descent (first red-black
// sweep from zero, residual, restriction) and the ascent (prolongation, black and red half-sweep, on level 0 the sums
// the CG step takes).
//
// What bounds such a level is not bytes but launches: run one operation per launch it costs six dependent launches of
// 3-7 us on a few hundred thousand cells or less. Here a block owns 8 x 8 x 16 cells, brings the region its results
// depend on (3 cells further on each side for the descent, 2 for the ascent) into registers and shared memory, and
// recomputes the neighbours' values there instead of waiting for another launch: 14 x 14 x 22 cells for 1024, four
// times the arithmetic of a level whose arithmetic is free. The operations, their operands and their order are those of
// nb_split.cu. The descent writes the smoothed iterate to a second vector (the level's residual vector, which nothing
// needs here), the ascent reads it there and writes the level's e, so no block reads what another one writes.
//
// Regions. Block (bi, bj, bk) owns planes i0 = 1 + 8 bi .. i0 + 7, rows j0 .. j0 + 7 and cells k = 16 bk + 1 .. + 16,
// the children of coarse cells I0 = 1 + 4 bi .. + 3, J0 .. + 3, K0 = 1 + 8 bk .. + 7. In one colour's rows the region
// holds elements 8 bk - 1 .. 8 bk + 9 (element m: cell k = 2m + q, q the row's parity), 11 of each colour. A value that
// would need a cell outside the region belongs to a cell no result depends on.
//
// Measured (B200): the 64^3 cavity's step (three such levels, 16 iterations) 1.77 -> 1.38 ms, two 128^3 FLIP steps (such
// levels from 66^3 down) 15.5 -> 13.5 ms, 256^3 (the same levels) 6.0 -> 5.9 ms. By level size, a whole step with the
// level's legs in launches of their operations / in one launch each (FP32, FP64; us): 34^3 994 / 845, 1035 / 902; 50^3
// 1243 / 1051, 1171 / 1021; 66^3 1259 / 1101, 1324 / 1148; 74^3 1443 / 1308, 1541 / 1509; 82^3 1710 / 1560, 1652 / 1609;
// 98^3 1737 / 1704, 1743 / 1894; 114^3 2034 / 2329, 2257 / 2810; 130^3 2053 / 2636, 2625 / 3559, where the recomputation
// costs more than the launches. Elongated levels gain too (122 x 122 x 18: 3741 / 3137, 3392 / 2843; 18 x 18 x 1002:
// 1325 / 1167, 2623 / 2450).
#include "nb_quad.cuh"

namespace nb
{

namespace
{

constexpr int kLegThreads = 256;
constexpr int kLegM = 11; // elements of a row's colour in a region

// A block's place; kHalo: cells of the region beyond the block's own along i and j
template <int kHalo> struct LegPos
{
    static constexpr int kR = 8 + 2 * kHalo;                     // planes, rows of the region
    static constexpr int kElems = kR * kR * kLegM;               // elements of one colour
    static constexpr int kPer = (kElems + kLegThreads - 1) / kLegThreads;
    static constexpr int kSI = kR * kLegM, kSJ = kLegM;          // strides in shared memory
    int i0, j0, m0; // first own plane and row; element 8 bk
    __device__ __forceinline__ LegPos()
    {
        i0 = 1 + 8 * (int)blockIdx.z;
        j0 = 1 + 8 * (int)blockIdx.y;
        m0 = 8 * (int)blockIdx.x;
    }
    // element idx of the region: its local plane and row, its global plane, row and element
    struct At
    {
        int li, lj, i, j, m;
    };
    __device__ __forceinline__ At at(int idx) const
    {
        At a;
        const int row = idx / kLegM;
        a.li = row / kR;
        a.lj = row - a.li * kR;
        a.i = i0 - kHalo + a.li;
        a.j = j0 - kHalo + a.lj;
        a.m = m0 - 1 + idx - row * kLegM;
        return a;
    }
};

// cell (i, j, element m of parity q) is one of the block's own
__device__ __forceinline__ bool OwnCell(int li, int lj, int halo, int m, int q, int m0)
{
    const int k = 2 * m + q;
    return li >= halo && li < halo + 8 && lj >= halo && lj < halo + 8 && k >= 2 * m0 + 1 && k <= 2 * m0 + 16;
}

} // namespace

// e (both colours) = the first red-black sweep from zero into tmp; rc = R (r - M e)
template <typename T>
__global__ void __launch_bounds__(kLegThreads) k_leg_down(LevelView v, LevelView cv, const uint8_t *__restrict__ du,
                                                          const uint8_t *__restrict__ pext, const T *__restrict__ r,
                                                          T *__restrict__ tmp, T *__restrict__ rc)
{
    using L = LegPos<3>;
    __shared__ T s0[L::kElems], s1[L::kElems];
    __shared__ T inv[32];
    const L P;
    const int t = threadIdx.x;
    const int hb = (int)v.sHalf;
    // what the layout fixes, before the wait
    unsigned d0[L::kPer], d1[L::kPer];
    int off[L::kPer]; // 32-bit: these levels are small
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        const bool in = idx < L::kElems && a.i >= 0 && a.i < v.Ny && a.j >= 0 && a.j < v.Nx && a.m >= 0 && a.m < v.sRS;
        off[n] = in ? a.i * v.sPS + a.j * v.sRS + a.m : -1;
        d0[n] = in ? du[off[n]] : 0u;
        d1[n] = in ? du[hb + off[n]] : 0u;
    }
    if (t < 32) inv[t] = t ? (T)1 / ((T)0.5 * (T)v.gamma * (T)t) : (T)0;
    // the coarse cell of a thread, and its red children's moved weights
    const int kk = t & 7, jj = (t >> 3) & 3, ii = t >> 5;
    const int K = 1 + P.m0 + kk, J = (P.j0 + 1) / 2 + jj, I = (P.i0 + 1) / 2 + ii;
    bool cOn = t < 128 && K <= cv.Nz - 2 && J <= cv.Nx - 2 && I <= cv.Ny - 2;
    if (cOn) cOn = (cv.code[(long long)I * cv.sI + (long long)J * cv.sJ + K] & CODE_UNKNOWN) != 0;
    unsigned px[2][2] = {};
    if (cOn)
#pragma unroll
        for (int ca = 0; ca < 2; ca++)
#pragma unroll
            for (int cb = 0; cb < 2; cb++)
            {
                const int a = 2 * I - 1 + ca, b = 2 * J - 1 + cb, q = (a + b) & 1;
                px[ca][cb] = pext[(long long)a * v.sPS + (long long)b * v.sRS + K - q] & 0x3Fu;
            }
    PdlWait();
    PdlTrigger();
    T r0[L::kPer], r1[L::kPer];
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        r0[n] = off[n] >= 0 ? r[off[n]] : (T)0;
        r1[n] = off[n] >= 0 ? r[hb + off[n]] : (T)0;
    }
    __syncthreads(); // inv
    const T g = (T)v.gamma, hg = (T)0.5 * (T)v.gamma;
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        if (idx < L::kElems) s0[idx] = r0[n] * inv[d0[n] & 0x7Fu];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        if (idx >= L::kElems || a.li < 1 || a.li > L::kR - 2 || a.lj < 1 || a.lj > L::kR - 2) continue;
        const T sh = ((a.i + a.j + 1) & 1) ? s0[idx + 1] : s0[idx - 1];
        const T s = ((s0[idx + L::kSI] + s0[idx - L::kSI]) + (s0[idx + L::kSJ] + s0[idx - L::kSJ])) + (s0[idx] + sh);
        s1[idx] = (r1[n] + g * s) * inv[d1[n] & 0x7Fu];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        if (idx >= L::kElems || a.li < 2 || a.li > L::kR - 3 || a.lj < 2 || a.lj > L::kR - 3) continue;
        const int q = (a.i + a.j) & 1;
        const T e0 = s0[idx];
        if (off[n] >= 0)
        {
            if (OwnCell(a.li, a.lj, 3, a.m, q, P.m0)) tmp[off[n]] = e0;
            if (OwnCell(a.li, a.lj, 3, a.m, q ^ 1, P.m0)) tmp[hb + off[n]] = s1[idx];
        }
        const T sh = q ? s1[idx + 1] : s1[idx - 1];
        const T s = ((s1[idx + L::kSI] + s1[idx - L::kSI]) + (s1[idx + L::kSJ] + s1[idx - L::kSJ])) + (s1[idx] + sh);
        // read by no other thread before the barrier: the red residual takes the red value's place
        s0[idx] = (d0[n] & 0x80u) ? r0[n] - (hg * (T)(d0[n] & 0x7Fu) * e0 - g * s) : (T)0;
    }
    __syncthreads();
    if (!cOn) return;
    // SplitRestrictPlane1's sums over fine planes 2I-2 .. 2I+1, rows 2J-2 .. 2J+1, red elements K-1 and K
    const T wt[4] = {(T)0.25, (T)0.75, (T)0.75, (T)0.25};
    T Tw[4], X[4];
#pragma unroll
    for (int da = 0; da < 4; da++)
    {
        Tw[da] = (T)0;
        X[da] = (T)0;
        const int a = 2 * I - 2 + da;
#pragma unroll
        for (int dj = 0; dj < 4; dj++)
        {
            const int b = 2 * J - 2 + dj, q = (a + b) & 1;
            const int at = (2 * ii + 2 + da) * L::kSI + (2 * jj + 2 + dj) * L::kSJ + kk + 1;
            const T lo = s0[at], hi = s0[at + 1];
            Tw[da] += wt[dj] * (q ? (T)0.75 * lo + (T)0.25 * hi : (T)0.25 * lo + (T)0.75 * hi);
            if ((da == 1 || da == 2) && (dj == 1 || dj == 2)) X[da] += (T)px[da - 1][dj - 1] * (q ? lo : hi);
        }
        X[da] *= (T)(1.0 / 64.0);
    }
    rc[VecIdx(cv, I, J, K)] =
        (((T)0.25 * Tw[0] + (T)0.75 * Tw[1]) + ((T)0.75 * Tw[2] + (T)0.25 * Tw[3])) + (X[1] + X[2]);
}

// e = tmp + P ec on the red cells, then a black and a red half-sweep. kDot (level 0): (sum r.e, sum e, sum r) into the
// scalar block of the iteration's parity.
template <typename T, bool kDot>
__global__ void __launch_bounds__(kLegThreads) k_leg_up(LevelView v, LevelView cv, const uint8_t *__restrict__ du,
                                                        const uint8_t *__restrict__ pext, const T *__restrict__ r,
                                                        const T *__restrict__ tmp, const T *__restrict__ ec,
                                                        T *__restrict__ e, Reducer R, const int *it, int baseEven,
                                                        int baseOdd)
{
    using L = LegPos<2>;
    constexpr int kC = 8, kCK = 12, kCoarse = kC * kC * kCK;
    __shared__ T s0[L::kElems], s1[L::kElems], c[kCoarse];
    __shared__ T inv[32];
    const L P;
    const int t = threadIdx.x;
    const int hb = (int)v.sHalf;
    unsigned d0[L::kPer], d1[L::kPer], px[L::kPer];
    int off[L::kPer]; // 32-bit: these levels are small
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        const bool in = idx < L::kElems && a.i >= 0 && a.i < v.Ny && a.j >= 0 && a.j < v.Nx && a.m >= 0 && a.m < v.sRS;
        off[n] = in ? a.i * v.sPS + a.j * v.sRS + a.m : -1;
        d0[n] = in ? du[off[n]] : 0u;
        d1[n] = in ? du[hb + off[n]] : 0u;
        px[n] = in ? pext[off[n]] : 0u;
    }
    if (t < 32) inv[t] = t ? (T)1 / ((T)0.5 * (T)v.gamma * (T)t) : (T)0;
    const int I0 = (P.i0 + 1) / 2, J0 = (P.j0 + 1) / 2;
    PdlWait();
    PdlTrigger();
    T r0[L::kPer], r1[L::kPer], e0[L::kPer];
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        e0[n] = off[n] >= 0 ? tmp[off[n]] : (T)0;
        r0[n] = off[n] >= 0 ? r[off[n]] : (T)0;
        r1[n] = off[n] >= 0 ? r[hb + off[n]] : (T)0;
    }
    // coarse cells I0-2 .. I0+5, J0-2 .. J0+5, m0-1 .. m0+10
#pragma unroll
    for (int n = 0; n < kCoarse / kLegThreads; n++)
    {
        const int idx = t + n * kLegThreads, row = idx / kCK;
        const int A = I0 - 2 + row / kC, B = J0 - 2 + row % kC, D = P.m0 - 1 + idx - row * kCK;
        const bool in = A >= 0 && A < cv.Ny && B >= 0 && B < cv.Nx && D >= 0 && D < cv.Nz;
        c[idx] = in ? ec[VecIdx(cv, A, B, D)] : (T)0;
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        if (idx >= L::kElems) continue;
        const typename L::At a = P.at(idx);
        T x = e0[n];
        if (px[n] & 0x80u)
        {
            // the parent's coarse plane and row, the other contributors', and k-cells m, m + 1 (SplitProlong's order)
            const int A = (a.i + 1) >> 1, A2 = A + ((a.i & 1) ? -1 : 1), B = (a.j + 1) >> 1, B2 = B + ((a.j & 1) ? -1 : 1);
            const int ck = a.m - P.m0 + 1;
            auto at = [&](int AA, int BB, int k) { return c[((AA - I0 + 2) * kC + (BB - J0 + 2)) * kCK + ck + k]; };
            T z[2];
#pragma unroll
            for (int k = 0; k < 2; k++)
            {
                const T yC = (T)0.75 * at(A, B, k) + (T)0.25 * at(A, B2, k);
                const T yO = (T)0.75 * at(A2, B, k) + (T)0.25 * at(A2, B2, k);
                z[k] = (T)0.75 * yC + (T)0.25 * yO;
            }
            const int q = (a.i + a.j) & 1;
            const T lohi = q ? (T)0.25 * z[0] + (T)0.75 * z[1] : (T)0.75 * z[0] + (T)0.25 * z[1];
            x += lohi + (T)(px[n] & 0x3Fu) * (T)(1.0 / 64.0) * at(A, B, q);
        }
        s0[idx] = x;
    }
    __syncthreads();
    const T g = (T)v.gamma;
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        if (idx >= L::kElems || a.li < 1 || a.li > L::kR - 2 || a.lj < 1 || a.lj > L::kR - 2) continue;
        const T sh = ((a.i + a.j + 1) & 1) ? s0[idx + 1] : s0[idx - 1];
        const T s = ((s0[idx + L::kSI] + s0[idx - L::kSI]) + (s0[idx + L::kSJ] + s0[idx - L::kSJ])) + (s0[idx] + sh);
        s1[idx] = (r1[n] + g * s) * inv[d1[n] & 0x7Fu];
    }
    __syncthreads();
    double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int n = 0; n < L::kPer; n++)
    {
        const int idx = t + n * kLegThreads;
        const typename L::At a = P.at(idx);
        if (idx >= L::kElems || off[n] < 0) continue;
        const int q = (a.i + a.j) & 1;
        if (OwnCell(a.li, a.lj, 2, a.m, q ^ 1, P.m0))
        {
            const T y = s1[idx];
            e[hb + off[n]] = y;
            if (kDot)
            {
                acc[0] += (double)r1[n] * (double)y;
                acc[1] += (double)y;
                acc[2] += (double)r1[n];
            }
        }
        if (OwnCell(a.li, a.lj, 2, a.m, q, P.m0))
        {
            const T sh = q ? s1[idx + 1] : s1[idx - 1];
            const T s = ((s1[idx + L::kSI] + s1[idx - L::kSI]) + (s1[idx + L::kSJ] + s1[idx - L::kSJ])) + (s1[idx] + sh);
            const T y = (r0[n] + g * s) * inv[d0[n] & 0x7Fu];
            e[off[n]] = y;
            if (kDot)
            {
                acc[0] += (double)r0[n] * (double)y;
                acc[1] += (double)y;
                acc[2] += (double)r0[n];
            }
        }
    }
    if (kDot) GridReduce<3>(R, acc, (*it & 1) ? baseOdd : baseEven);
}

// blocks over the level's coarse cells: every own cell is a child of one of them
static dim3 LegGrid(const LevelView &cv)
{
    return dim3((unsigned)((cv.Nz - 2 + 7) / 8), (unsigned)((cv.Nx - 2 + 3) / 4), (unsigned)((cv.Ny - 2 + 3) / 4));
}

template <typename T>
void LaunchLegDown(const LevelView &v, const LevelView &cv, const uint8_t *du, const uint8_t *pext, const T *r, T *tmp,
                   T *rc, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(k_leg_down<T>, LegGrid(cv), dim3(kLegThreads), 0, st, v, cv, du, pext, r, tmp, rc);
}

template <typename T>
void LaunchLegUp(const LevelView &v, const LevelView &cv, const uint8_t *du, const uint8_t *pext, const T *r,
                 const T *tmp, const T *ec, T *e, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(k_leg_up<T, false>, LegGrid(cv), dim3(kLegThreads), 0, st, v, cv, du, pext, r, tmp, ec, e, Reducer{},
              (const int *)nullptr, 0, 0);
}

template <typename T>
void LaunchLegUpDot(const LevelView &v, const LevelView &cv, const uint8_t *du, const uint8_t *pext, const T *r,
                    const T *tmp, const T *ec, T *e, const Reducer &R, const int *it, int baseEven, int baseOdd,
                    cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(k_leg_up<T, true>, SumGrid(R, LegGrid(cv)), dim3(kLegThreads), 0, st, v, cv, du, pext, r, tmp, ec, e, R, it,
              baseEven, baseOdd);
}

#define NB_INST(T)                                                                                                 \
    template void LaunchLegDown<T>(const LevelView &, const LevelView &, const uint8_t *, const uint8_t *,         \
                                   const T *, T *, T *, cudaStream_t);                                             \
    template void LaunchLegUp<T>(const LevelView &, const LevelView &, const uint8_t *, const uint8_t *,           \
                                 const T *, const T *, const T *, T *, cudaStream_t);                              \
    template void LaunchLegUpDot<T>(const LevelView &, const LevelView &, const uint8_t *, const uint8_t *,        \
                                    const T *, const T *, const T *, T *, const Reducer &, const int *, int, int,  \
                                    cudaStream_t);
NB_INST(float)
NB_INST(double)
#undef NB_INST

} // namespace nb
