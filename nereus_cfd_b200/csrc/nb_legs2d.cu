// The two legs of the V-cycle on a 2D level, one kernel each, T = float or double, uniform or stretched: the descent
// (the red-black sweeps from zero, the residual, its restriction) and the ascent (prolongation, the black-red sweeps, on
// level 0 the sums the CG step takes).
//
// A 2D level holds at most a million cells or so and mostly far fewer: its time is launches and their latency, seven of
// them a level. Here a block owns 16 x 32 cells, brings them and a halo into shared memory and recomputes the
// neighbours' values there instead of waiting for another launch: with one sweep 22 x 38 cells for the descent and
// 20 x 36 for the ascent. The descent writes the smoothed iterate to the level's residual vector, the ascent reads it
// there and writes the level's e, so no block reads what another one writes.
//
// The values are those of the per-cell kernels (nb_kernels.cu): the same coefficients (the level's FP32 tables; 1 on a
// uniform level), diagonal (kept per cell, once per layout), sums in the same order and division, so that a solve ends
// where it ended with a launch per operation. Reciprocals and sums by pairs instead took 6% off the step and
// moved the pressure by up to 3e-7 of itself (FP32 rounding, carried through a solve to 1e-8).
//
// Measured (B200): the 128^2 closed box's step in mixed precision to 1e-10 (13 iterations, two such levels) 1.03 -> 0.79 ms
// with the ring replay in one launch. No line in size: a step around a disc to 1e-10 with the per-cell kernels / with the
// legs (mixed, FP64; ms) 64^2 1.02 / 0.84, 0.91 / 0.74; 256^2 1.59 / 1.15, 1.51 / 1.13; 1024^2 4.86 / 3.42, 4.36 / 3.30;
// 2048^2 14.1 / 10.3, 12.8 / 10.0; 3900^2 71.4 / 48.7, 56.7 / 41.0.
#include "nb_kernels.h"

namespace nb
{

namespace
{

constexpr int kThreads2 = 256;
constexpr int kOwnI = 16, kOwnJ = 32; // the block's own fine cells: 8 x 16 coarse cells' children

// a thread block's region of the level: kHalo cells beyond its own on every side
template <int kHalo> struct Region2
{
    static constexpr int kR = kOwnI + 2 * kHalo, kC = kOwnJ + 2 * kHalo, kN = kR * kC;
    int i0, j0; // the region's first cell (may lie outside the grid)
    __device__ __forceinline__ Region2()
    {
        i0 = 1 + kOwnI * (int)blockIdx.y - kHalo;
        j0 = 1 + kOwnJ * (int)blockIdx.x - kHalo;
    }
};

// the region's 1D tables: Width and 1/FaceGap (FP32, as LevelCoefs reads them) along both axes, 1 on a uniform level
template <typename T, int kR, int kC> struct Tables2
{
    T wy[kR], gy[kR + 1], wx[kC], gx[kC + 1]; // g[n]: the face below cell n of the region
};

template <typename T, int kR, int kC>
__device__ __forceinline__ void LoadTables(const LevelView &v, int i0, int j0, Tables2<T, kR, kC> &s)
{
    auto entry = [](const float *tab, int n, int last) { return (T)tab[n < 0 ? 0 : (n > last ? last : n)]; };
    for (int n = threadIdx.x; n <= kR; n += kThreads2)
    {
        if (n < kR) s.wy[n] = v.stretched ? entry(v.w32[1], i0 + n + 1, v.Ny + 1) : (T)1;
        s.gy[n] = v.stretched ? entry(v.ig32[1], i0 + n, v.Ny) : (T)1;
    }
    for (int n = threadIdx.x; n <= kC; n += kThreads2)
    {
        if (n < kC) s.wx[n] = v.stretched ? entry(v.w32[0], j0 + n + 1, v.Nx + 1) : (T)1;
        s.gx[n] = v.stretched ? entry(v.ig32[0], j0 + n, v.Nx) : (T)1;
    }
}

// the coefficient-weighted sum of a cell's neighbours, in MaskedSum's order (a neighbour that is no unknown holds zero)
template <typename T, int kR, int kC>
__device__ __forceinline__ T Sum2(const Tables2<T, kR, kC> &s, const T *e, int li, int lj)
{
    const T *p = e + li * kC + lj;
    const T wx = s.wx[lj], wy = s.wy[li];
    const T c0 = wx * s.gy[li + 1], c1 = wx * s.gy[li], c2 = wy * s.gx[lj + 1], c3 = wy * s.gx[lj];
    T x = c0 * p[kC];
    x += c1 * p[-kC];
    x += c2 * p[1];
    x += c3 * p[-1];
    return x;
}

// a sweep's new value: rhs / diagonal (zero off the unknowns and at an unknown without neighbours)
template <typename T> __device__ __forceinline__ T OverDiag(T rhs, T d) { return d != (T)0 ? rhs / d : (T)0; }

// Runs f(li, lj) over the cells of the colour in the region shrunk by `m` on every side, then the barrier.
template <int kR, int kC, typename F>
__device__ __forceinline__ void ForColour(int i0, int j0, int m, int colour, F f)
{
    const int rows = kR - 2 * m, half = (kC - 2 * m) / 2; // kC is even
    for (int t = threadIdx.x; t < rows * half; t += kThreads2)
    {
        const int a = t / half, li = m + a;
        const int lj = m + 2 * (t - a * half) + ((i0 + li + j0 + m + colour) & 1);
        f(li, lj);
    }
    __syncthreads();
}

__device__ __forceinline__ bool InGrid(const LevelView &v, int i, int j)
{
    return i >= 0 && i < v.Ny && j >= 0 && j < v.Nx;
}

} // namespace

// per layout: the diagonal of every unknown as the per-cell kernels of the solver's precision form it (zero elsewhere),
// and the weights the transfers move off SOLID coarse contributors (0x80 | 64ths at an unknown)
template <typename T>
__global__ void __launch_bounds__(256) k_build_2d(LevelView v, LevelView cv, double *__restrict__ dg,
                                                  uint8_t *__restrict__ ext)
{
    const int c = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= (int)v.cells) return;
    const unsigned code = v.code[c];
    T d = (T)0;
    unsigned moved = 0;
    if (code & CODE_UNKNOWN)
    {
        const int i = c / v.Nx, j = c - i * v.Nx;
        T cq[6];
        CodeStencil<T>(v, i, j, 0, c, code, cq, d);
        const int I = (i + 1) >> 1, J = (j + 1) >> 1, si = (i & 1) ? -1 : 1, sj = (j & 1) ? -1 : 1;
        moved = 0x80u;
        for (int q = 1; q < 4; q++)
        {
            const int di = q & 1, dj = q >> 1;
            if (cv.types[(long long)(I + di * si) * cv.sI + J + dj * sj] == SOLID)
                moved += 4u * (di ? 1u : 3u) * (dj ? 1u : 3u);
        }
    }
    dg[c] = (double)d;
    ext[c] = (uint8_t)moved;
}

void LaunchBuild2D(const LevelView &v, const LevelView &cv, int elemBytes, double *dg, uint8_t *ext, cudaStream_t st)
{
    const unsigned blocks = (unsigned)((v.cells + 255) / 256);
    NB_COUNT_LAUNCH();
    if (elemBytes == 8) k_build_2d<double><<<blocks, 256, 0, st>>>(v, cv, dg, ext);
    else k_build_2d<float><<<blocks, 256, 0, st>>>(v, cv, dg, ext);
}

// tmp = kS red-black sweeps from zero; rc = R (r - M tmp)
template <typename T, int kS>
__global__ void __launch_bounds__(kThreads2) k_leg2_down(LevelView v, LevelView cv, const uint8_t *__restrict__ ext,
                                                         const T *__restrict__ r, T *__restrict__ tmp,
                                                         T *__restrict__ rc)
{
    constexpr int kHalo = 2 * kS + 1;
    using G = Region2<kHalo>;
    __shared__ T sr[G::kN], sd[G::kN], se[G::kN];
    __shared__ Tables2<T, G::kR, G::kC> tab;
    const G P;
    LoadTables<T, G::kR, G::kC>(v, P.i0, P.j0, tab);
    for (int t = threadIdx.x; t < G::kN; t += kThreads2)
    {
        const int i = P.i0 + t / G::kC, j = P.j0 + t % G::kC;
        sd[t] = InGrid(v, i, j) ? (T)v.dg[i * v.Nx + j] : (T)0;
    }
    PdlWait();
    PdlTrigger();
    for (int t = threadIdx.x; t < G::kN; t += kThreads2)
    {
        const int i = P.i0 + t / G::kC, j = P.j0 + t % G::kC;
        const T x = InGrid(v, i, j) ? r[i * v.Nx + j] : (T)0;
        sr[t] = x;
        se[t] = OverDiag(x, sd[t]); // the red half from zero (the black values are replaced unread)
    }
    __syncthreads();
#pragma unroll
    for (int h = 1; h < 2 * kS; h++)
        ForColour<G::kR, G::kC>(P.i0, P.j0, h, h & 1, [&](int li, int lj) {
            const int t = li * G::kC + lj;
            se[t] = OverDiag(sr[t] + Sum2<T, G::kR, G::kC>(tab, se, li, lj), sd[t]);
        });
    for (int t = threadIdx.x; t < kOwnI * kOwnJ; t += kThreads2)
    {
        const int li = kHalo + t / kOwnJ, lj = kHalo + t % kOwnJ, i = P.i0 + li, j = P.j0 + lj;
        if (i <= v.Ny - 2 && j <= v.Nx - 2) tmp[i * v.Nx + j] = se[li * G::kC + lj];
    }
    // the residual, over r (of both colours: the black one is what the division's rounding leaves, as in the per-cell
    // kernels)
#pragma unroll
    for (int colour = 0; colour < 2; colour++)
        ForColour<G::kR, G::kC>(P.i0, P.j0, 2 * kS, colour, [&](int li, int lj) {
            const int t = li * G::kC + lj, i = P.i0 + li, j = P.j0 + lj;
            T x = (T)0;
            if (InGrid(v, i, j) && (v.code[i * v.Nx + j] & CODE_UNKNOWN))
                x = sr[t] - (sd[t] * se[t] - Sum2<T, G::kR, G::kC>(tab, se, li, lj));
            sr[t] = x;
        });
    if (threadIdx.x >= (kOwnI / 2) * (kOwnJ / 2)) return;
    const int ii = threadIdx.x / (kOwnJ / 2), jj = threadIdx.x % (kOwnJ / 2);
    const int I = (P.i0 + kHalo + 1) / 2 + ii, J = (P.j0 + kHalo + 1) / 2 + jj;
    if (I > cv.Ny - 2 || J > cv.Nx - 2 || !(cv.code[I * cv.Nx + J] & CODE_UNKNOWN)) return;
    const T wt[4] = {(T)0.25, (T)0.75, (T)0.75, (T)0.25};
    T acc = (T)0;
    // fine cell (2I - 2 + di, 2J - 2 + dj): I, J are the own region's (ii, jj)-th, whose first child is its first cell
    const T *x = sr + (kHalo - 1 + 2 * ii) * G::kC + kHalo - 1 + 2 * jj;
#pragma unroll
    for (int di = 0; di < 4; di++)
#pragma unroll
        for (int dj = 0; dj < 4; dj++) acc += wt[di] * wt[dj] * x[di * G::kC + dj];
#pragma unroll
    for (int di = 1; di < 3; di++)
#pragma unroll
        for (int dj = 1; dj < 3; dj++)
        {
            const int i = 2 * I - 2 + di, j = 2 * J - 2 + dj;
            const unsigned m = InGrid(v, i, j) ? ext[i * v.Nx + j] & 0x3Fu : 0u;
            if (m) acc += (T)m * (T)(1.0 / 64.0) * x[di * G::kC + dj];
        }
    rc[I * cv.Nx + J] = acc;
}

// e = kS black-red sweeps after tmp + P ec. kDot (level 0): (sum r.e, sum e, sum r) into the scalar block of the
// iteration's parity.
template <typename T, int kS, bool kDot>
__global__ void __launch_bounds__(kThreads2) k_leg2_up(LevelView v, LevelView cv, const uint8_t *__restrict__ ext,
                                                       const T *__restrict__ r, const T *__restrict__ tmp,
                                                       const T *__restrict__ ec, T *__restrict__ e, Reducer R,
                                                       const int *it, int baseEven, int baseOdd)
{
    constexpr int kHalo = 2 * kS;
    using G = Region2<kHalo>;
    constexpr int kCR = kOwnI / 2 + 2 * kS + 2, kCC = kOwnJ / 2 + 2 * kS + 2; // coarse cells the region's come from
    __shared__ T sr[G::kN], sd[G::kN], se[G::kN], sc[kCR * kCC];
    __shared__ Tables2<T, G::kR, G::kC> tab;
    const G P;
    LoadTables<T, G::kR, G::kC>(v, P.i0, P.j0, tab);
    for (int t = threadIdx.x; t < G::kN; t += kThreads2)
    {
        const int i = P.i0 + t / G::kC, j = P.j0 + t % G::kC;
        sd[t] = InGrid(v, i, j) ? (T)v.dg[i * v.Nx + j] : (T)0;
    }
    const int A0 = (P.i0 + kHalo + 1) / 2 - kS - 1, B0 = (P.j0 + kHalo + 1) / 2 - kS - 1;
    PdlWait();
    PdlTrigger();
    for (int t = threadIdx.x; t < G::kN; t += kThreads2)
    {
        const int i = P.i0 + t / G::kC, j = P.j0 + t % G::kC;
        const bool in = InGrid(v, i, j);
        sr[t] = in ? r[i * v.Nx + j] : (T)0;
        se[t] = in ? tmp[i * v.Nx + j] : (T)0;
    }
    for (int t = threadIdx.x; t < kCR * kCC; t += kThreads2)
    {
        const int A = A0 + t / kCC, B = B0 + t % kCC;
        sc[t] = InGrid(cv, A, B) ? ec[A * cv.Nx + B] : (T)0;
    }
    __syncthreads();
    // the coarse correction on the red cells (the black half that follows replaces the black values unread)
    ForColour<G::kR, G::kC>(P.i0, P.j0, 0, 0, [&](int li, int lj) {
        const int i = P.i0 + li, j = P.j0 + lj;
        const unsigned x = InGrid(v, i, j) ? ext[i * v.Nx + j] : 0u;
        if (!(x & 0x80u)) return;
        const int si = (i & 1) ? -kCC : kCC, sj = (j & 1) ? -1 : 1;
        const T *p = sc + (((i + 1) >> 1) - A0) * kCC + ((j + 1) >> 1) - B0;
        T acc = (T)0;
        acc += (T)0.5625 * p[0];
        acc += (T)0.1875 * p[sj];
        acc += (T)0.1875 * p[si];
        acc += (T)0.0625 * p[si + sj];
        se[li * G::kC + lj] += acc + (T)(x & 0x3Fu) * (T)(1.0 / 64.0) * p[0];
    });
#pragma unroll
    for (int h = 1; h <= 2 * kS; h++)
        ForColour<G::kR, G::kC>(P.i0, P.j0, h, h & 1, [&](int li, int lj) {
            const int t = li * G::kC + lj;
            se[t] = OverDiag(sr[t] + Sum2<T, G::kR, G::kC>(tab, se, li, lj), sd[t]);
        });
    double acc[3] = {0.0, 0.0, 0.0};
    for (int t = threadIdx.x; t < kOwnI * kOwnJ; t += kThreads2)
    {
        const int li = kHalo + t / kOwnJ, lj = kHalo + t % kOwnJ, i = P.i0 + li, j = P.j0 + lj;
        if (i > v.Ny - 2 || j > v.Nx - 2) continue;
        const T y = se[li * G::kC + lj];
        e[i * v.Nx + j] = y;
        if (kDot)
        {
            const double rr = (double)sr[li * G::kC + lj];
            acc[0] += rr * (double)y;
            acc[1] += (double)y;
            acc[2] += rr;
        }
    }
    if (kDot) GridReduce<3>(R, acc, (*it & 1) ? baseOdd : baseEven);
}

static dim3 Leg2Grid(const LevelView &v)
{
    return dim3((unsigned)((v.Nx - 2 + kOwnJ - 1) / kOwnJ), (unsigned)((v.Ny - 2 + kOwnI - 1) / kOwnI));
}

long long Leg2SumBlocks(const LevelView &v)
{
    const dim3 g = Leg2Grid(v);
    return (long long)g.x * g.y;
}

template <typename T>
void LaunchLeg2Down(const LevelView &v, const LevelView &cv, const uint8_t *ext, const T *r, T *tmp, T *rc, int sweeps,
                    cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    if (sweeps == 1) LaunchPdl(k_leg2_down<T, 1>, Leg2Grid(v), dim3(kThreads2), 0, st, v, cv, ext, r, tmp, rc);
    else LaunchPdl(k_leg2_down<T, 2>, Leg2Grid(v), dim3(kThreads2), 0, st, v, cv, ext, r, tmp, rc);
}

template <typename T>
void LaunchLeg2Up(const LevelView &v, const LevelView &cv, const uint8_t *ext, const T *r, const T *tmp, const T *ec,
                  T *e, int sweeps, bool dot, const Reducer &R, const int *it, int baseEven, int baseOdd,
                  cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    auto go = [&](auto kernel) {
        LaunchPdl(kernel, dot ? SumGrid(R, Leg2Grid(v)) : Leg2Grid(v), dim3(kThreads2), 0, st, v, cv, ext, r, tmp, ec, e, R,
                  it, baseEven, baseOdd);
    };
    if (sweeps == 1) dot ? go(k_leg2_up<T, 1, true>) : go(k_leg2_up<T, 1, false>);
    else dot ? go(k_leg2_up<T, 2, true>) : go(k_leg2_up<T, 2, false>);
}

#define NB_INST(T)                                                                                                 \
    template void LaunchLeg2Down<T>(const LevelView &, const LevelView &, const uint8_t *, const T *, T *, T *,    \
                                    int, cudaStream_t);                                                            \
    template void LaunchLeg2Up<T>(const LevelView &, const LevelView &, const uint8_t *, const T *, const T *,     \
                                  const T *, T *, int, bool, const Reducer &, const int *, int, int, cudaStream_t);
NB_INST(float)
NB_INST(double)
#undef NB_INST

} // namespace nb
