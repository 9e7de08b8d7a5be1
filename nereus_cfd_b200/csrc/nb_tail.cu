// The coarse end of the multigrid V-cycle in one thread block: every level from `tailStart` down (at most a few
// thousand cells each) lives in shared memory, and the block runs their pre-smoothing, residual, restriction,
// coarsest sweeps, prolongation and post-smoothing back to back. It reads the restricted residual of the first tail
// level from global memory and writes that level's correction back; the finer levels' kernels on either side are
// unchanged. The operations are the ones of nb_kernels.cu (same stencil, transfers and colour order), so the
// V-cycle stays the same symmetric operator.
//
// What costs time here is latency, not bytes: each phase (one colour of a sweep, a residual, a transfer) is a short
// loop over a level's unknowns followed by a barrier. So
// - what a layout fixes is built once per layout (k_tail_lists) in the order it has in shared memory and only copied
//   in, 16 bytes at a time, before the dependent-launch wait: the per-colour lists of unknowns, the diagonal's
//   half-units (uniform) or the codes and types (stretched), and the weights the transfers move off SOLID cells;
// - a uniform level sums its six neighbours unmasked (every vector is zero off the unknowns) and divides through a
//   per-level reciprocal table of the diagonal's half-units;
// - a thread keeps its red and its black cell's index, right-hand side and stencil in registers across a level's
//   sweeps and residual, where a level has at most one unknown of each colour per thread (all but the first levels
//   of unusually large coarse ends); a half-sweep then waits for its six neighbours only;
// - the levels with at most 32 unknowns of each colour (the last two or three) run in warp 0 alone, with __syncwarp
//   between their phases instead of a block-wide barrier.
// Against a form that prepared the lists alone, decoded its cells and read its stencil again in every phase, this took
// 10 us off each V-cycle of a 64^3 box (of 120), 8 off one of a 2D 128^2 box (of 86) and 21 off one of the stretched
// FP64 cylinder (of 410; B200).
#include "nb_kernels.h"

#include <cstring>
#include <mutex>
#include <set>

namespace nb
{

// threads of the block: one per unknown of a colour on the usual coarse ends (a first level of at most 2048 cells)
constexpr int kTailThreads = 256, kTailThreadsBig = 512;

template <typename T> struct TailLevel
{
    LevelView v;
    unsigned off;     // byte offset of the level's arrays in shared memory
    unsigned listOff; // 4-byte offset of the level's prepared data in the global array
    unsigned vecs; // vectors in shared memory: r, e and, but for the coarsest level, res
};

template <typename T> struct TailArgs
{
    TailLevel<T> lv[kMaxTailLevels];
    int nlev;
    const T *rIn; // residual of the first tail level (global)
    T *eOut;      // its correction (global)
    int pre, post, coarseSweeps;
    const unsigned *lists; // per level: its prepared data (PrepBytes)
    const int *counts;     // [level][colour] unknowns
};

__host__ __device__ inline unsigned Pad16(unsigned b) { return (b + 15u) / 16u * 16u; }

// A level's prepared data, the same bytes in global and shared memory: the list of its unknowns (4 bytes each, packed
// i << 20 | j << 10 | k: red ones from the front, black ones from the back), then three byte arrays: the diagonal's
// half-units, the transfer weights and nothing (uniform), or the codes, the transfer weights and the types (stretched).
__host__ __device__ inline unsigned PrepBytes(long long cells)
{
    return Pad16((unsigned)cells * 4u) + 3u * Pad16((unsigned)cells);
}

// The level's arrays in shared memory: r, e and, but for the coarsest level, res (T), then its prepared data, each padded
// to 16 bytes.
template <typename T> __host__ __device__ inline unsigned LevelBytes(long long cells, bool last)
{
    return (last ? 2u : 3u) * Pad16((unsigned)(cells * sizeof(T))) + PrepBytes(cells);
}

template <typename T> struct SmemLevel
{
    int sI, sJ, cells;
    int Nx, Ny, Nz;
    T *r, *e, *res;
    unsigned *list;      // red [0, nRed), black [cells - nBlack, cells)
    const uint8_t *unit; // uniform: 0x80 | diagonal half-units at an unknown, 0 elsewhere; stretched: the codes
    const uint8_t *ext;  // 0x80 | 64ths of weight the transfers move onto the parent, at an unknown
    const uint8_t *types; // stretched
    int nRed, nBlack;
    T g, hg;             // gamma, gamma / 2 (uniform)
    const double *inv;   // 1 / (gamma/2 * units), entry 0 = 0
    const LevelView *v;  // the spacing tables (stretched)
};

__device__ __forceinline__ void Unpack(unsigned x, int &i, int &j, int &k)
{
    i = (int)(x >> 20);
    j = (int)((x >> 10) & 1023u);
    k = (int)(x & 1023u);
}

template <typename T> __device__ __forceinline__ SmemLevel<T> Bind(const TailLevel<T> &tl, unsigned char *smem)
{
    SmemLevel<T> s;
    s.v = &tl.v;
    s.sI = (int)tl.v.sI;
    s.sJ = (int)tl.v.sJ;
    s.cells = (int)tl.v.cells;
    s.Nx = tl.v.Nx;
    s.Ny = tl.v.Ny;
    s.Nz = tl.v.Nz;
    s.g = (T)tl.v.gamma;
    s.hg = (T)0.5 * (T)tl.v.gamma;
    const unsigned a = Pad16((unsigned)(s.cells * sizeof(T))), b = Pad16((unsigned)s.cells);
    unsigned char *base = smem + tl.off;
    s.r = (T *)base;
    s.e = (T *)(base + a);
    s.res = (T *)(base + 2 * a);
    s.list = (unsigned *)(base + tl.vecs * a);
    s.unit = base + tl.vecs * a + Pad16((unsigned)s.cells * 4u);
    s.ext = s.unit + b;
    s.types = s.ext + b;
    s.nRed = s.nBlack = 0;
    s.inv = nullptr;
    return s;
}

// the t-th unknown of the given colour (0 red, 1 black, 2 both: red then black)
template <typename T> __device__ __forceinline__ unsigned ListAt(const SmemLevel<T> &L, int colour, int t)
{
    if (colour == 0) return L.list[t];
    if (colour == 1) return L.list[L.cells - 1 - t];
    return t < L.nRed ? L.list[t] : L.list[L.cells - 1 - (t - L.nRed)];
}

template <typename T> __device__ __forceinline__ int ListLen(const SmemLevel<T> &L, int colour)
{
    return colour == 0 ? L.nRed : (colour == 1 ? L.nBlack : L.nRed + L.nBlack);
}

// A phase runs over the whole block (kWarp false) or over warp 0 alone (kWarp true), and ends with the matching
// barrier.
template <bool kWarp> __device__ __forceinline__ int PhaseStart()
{
    return kWarp ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
}
template <bool kWarp> __device__ __forceinline__ int PhaseStride() { return kWarp ? 32 : (int)blockDim.x; }
template <bool kWarp> __device__ __forceinline__ void PhaseSync()
{
    if (kWarp) __syncwarp();
    else __syncthreads();
}

// One unknown of a level and its stencil
template <typename T, bool k3D, bool kSt> struct Cell
{
    int c;
    T r;
    unsigned b;             // uniform: the half-units byte; stretched: the code
    T inv;                  // uniform: 1 / diagonal
    T cq[kSt ? 6 : 1], diag; // stretched
};

template <typename T, bool k3D, bool kSt>
__device__ __forceinline__ Cell<T, k3D, kSt> LoadCell(const SmemLevel<T> &L, unsigned packed)
{
    Cell<T, k3D, kSt> o;
    int i, j, k;
    Unpack(packed, i, j, k);
    o.c = i * L.sI + j * L.sJ + k;
    o.r = L.r[o.c];
    o.b = L.unit[o.c];
    if constexpr (!kSt) o.inv = (T)L.inv[o.b & 0x7Fu];
    else
    {
        LevelView v = *L.v;
        v.types = L.types;
        CodeStencil<T>(v, i, j, k, o.c, o.b, o.cq, o.diag);
    }
    return o;
}

// the plain sum of a cell's neighbours on a uniform level (vectors are zero off the unknowns)
template <typename T, bool k3D> __device__ __forceinline__ T NbrSum(const SmemLevel<T> &L, const T *e, int c)
{
    const T s = (e[c + L.sI] + e[c - L.sI]) + (e[c + L.sJ] + e[c - L.sJ]);
    return k3D ? s + (e[c + 1] + e[c - 1]) : s;
}

template <typename T, bool k3D, bool kSt>
__device__ __forceinline__ void SmoothCell(const SmemLevel<T> &L, const Cell<T, k3D, kSt> &o, bool first)
{
    const int c = o.c;
    T rhs = o.r;
    if constexpr (!kSt)
    {
        if (!first) rhs += L.g * NbrSum<T, k3D>(L, L.e, c);
        L.e[c] = rhs * o.inv;
    }
    else
    {
        if (!first)
        {
            if (o.b & 1u) rhs += o.cq[0] * L.e[c + L.sI];
            if (o.b & 2u) rhs += o.cq[1] * L.e[c - L.sI];
            if (o.b & 4u) rhs += o.cq[2] * L.e[c + L.sJ];
            if (o.b & 8u) rhs += o.cq[3] * L.e[c - L.sJ];
            if (o.b & 16u) rhs += o.cq[4] * L.e[c + 1];
            if (o.b & 32u) rhs += o.cq[5] * L.e[c - 1];
        }
        L.e[c] = o.diag != (T)0 ? rhs / o.diag : (T)0;
    }
}

template <typename T, bool k3D, bool kSt>
__device__ __forceinline__ void ResidualCell(const SmemLevel<T> &L, const Cell<T, k3D, kSt> &o)
{
    const int c = o.c;
    if constexpr (!kSt)
    {
        // the products' rounding written out: contracted another way, the FP32 V-cycle's corrections (and with them a
        // mixed solve's last digits, 1e-8 to 3e-7 of the pressure) would differ from those of the per-cell kernels
        const T M = fma(-L.g, NbrSum<T, k3D>(L, L.e, c), L.hg * (T)(o.b & 0x7Fu) * L.e[c]);
        L.res[c] = o.r - M;
    }
    else
    {
        T s = o.diag * L.e[c];
        if (o.b & 1u) s -= o.cq[0] * L.e[c + L.sI];
        if (o.b & 2u) s -= o.cq[1] * L.e[c - L.sI];
        if (o.b & 4u) s -= o.cq[2] * L.e[c + L.sJ];
        if (o.b & 8u) s -= o.cq[3] * L.e[c - L.sJ];
        if (o.b & 16u) s -= o.cq[4] * L.e[c + 1];
        if (o.b & 32u) s -= o.cq[5] * L.e[c - 1];
        L.res[c] = o.r - s;
    }
}

// Sweeps of a level by one thread's cells: `fwd` red-black pairs (the first from a zero iterate where zero is set),
// then `bwd` black-red pairs, then the residual where res is set.
template <typename T, bool k3D, bool kSt, bool kWarp>
__device__ __forceinline__ void TSweeps(const SmemLevel<T> &L, int fwd, int bwd, bool zero, bool res)
{
    const int t0 = PhaseStart<kWarp>(), stride = PhaseStride<kWarp>();
    if (L.nRed <= stride && L.nBlack <= stride)
    {
        const bool hasR = t0 < L.nRed, hasB = t0 < L.nBlack;
        Cell<T, k3D, kSt> red{}, black{};
        if (hasR) red = LoadCell<T, k3D, kSt>(L, ListAt(L, 0, t0));
        if (hasB) black = LoadCell<T, k3D, kSt>(L, ListAt(L, 1, t0));
        for (int s = 0; s < fwd; s++)
        {
            if (hasR) SmoothCell(L, red, zero && s == 0);
            PhaseSync<kWarp>();
            if (hasB) SmoothCell(L, black, false);
            PhaseSync<kWarp>();
        }
        for (int s = 0; s < bwd; s++)
        {
            if (hasB) SmoothCell(L, black, false);
            PhaseSync<kWarp>();
            if (hasR) SmoothCell(L, red, false);
            PhaseSync<kWarp>();
        }
        if (res)
        {
            if (hasR) ResidualCell(L, red);
            if (hasB) ResidualCell(L, black);
            PhaseSync<kWarp>();
        }
        return;
    }
    auto half = [&](int colour, bool first) {
        const int n = ListLen(L, colour);
        for (int t = t0; t < n; t += stride) SmoothCell(L, LoadCell<T, k3D, kSt>(L, ListAt(L, colour, t)), first);
        PhaseSync<kWarp>();
    };
    for (int s = 0; s < fwd; s++)
    {
        half(0, zero && s == 0);
        half(1, false);
    }
    for (int s = 0; s < bwd; s++)
    {
        half(1, false);
        half(0, false);
    }
    if (res)
    {
        const int n = ListLen(L, 2);
        for (int t = t0; t < n; t += stride) ResidualCell(L, LoadCell<T, k3D, kSt>(L, ListAt(L, 2, t)));
        PhaseSync<kWarp>();
    }
}

// 64ths of moved weight at fine cell c, as a weight
template <typename T> __device__ __forceinline__ T Moved(const SmemLevel<T> &F, int c)
{
    return (T)(F.ext[c] & 0x3Fu) * (T)(1.0 / 64.0);
}

template <typename T, bool k3D, bool kWarp> __device__ void TRestrict(const SmemLevel<T> &F, const SmemLevel<T> &C)
{
    const int n = ListLen(C, 2);
    const T wt[4] = {(T)0.25, (T)0.75, (T)0.75, (T)0.25};
    for (int t = PhaseStart<kWarp>(); t < n; t += PhaseStride<kWarp>())
    {
        int I, J, K;
        Unpack(ListAt(C, 2, t), I, J, K);
        T acc = (T)0;
#pragma unroll
        for (int di = 0; di < 4; di++)
        {
            const int a = 2 * I - 2 + di;
            if (a > F.Ny - 1) continue;
#pragma unroll
            for (int dj = 0; dj < 4; dj++)
            {
                const int b = 2 * J - 2 + dj;
                if (b > F.Nx - 1) continue;
                const int rowBase = a * F.sI + b * F.sJ;
                const T wij = wt[di] * wt[dj];
                if (k3D)
                {
                    T s = (T)0;
#pragma unroll
                    for (int dk = 0; dk < 4; dk++)
                    {
                        const int d = 2 * K - 2 + dk;
                        if (d <= F.Nz - 1) s += wt[dk] * F.res[rowBase + d];
                    }
                    acc += wij * s;
                }
                else
                    acc += wij * F.res[rowBase];
            }
        }
        // the children also carry the weight the prolongation moved off their SOLID coarse contributors
#pragma unroll
        for (int ci = 0; ci < 2; ci++)
#pragma unroll
            for (int cj = 0; cj < 2; cj++)
#pragma unroll
                for (int ck = 0; ck < (k3D ? 2 : 1); ck++)
                {
                    const int a = 2 * I - 1 + ci, b = 2 * J - 1 + cj, d = k3D ? 2 * K - 1 + ck : 0;
                    if (a > F.Ny - 2 || b > F.Nx - 2 || (k3D && d > F.Nz - 2)) continue;
                    const int c = a * F.sI + b * F.sJ + d;
                    const T extra = Moved(F, c);
                    if (extra != (T)0) acc += extra * F.res[c];
                }
        C.r[I * C.sI + J * C.sJ + K] = acc;
    }
    PhaseSync<kWarp>();
}

template <typename T, bool k3D, bool kWarp> __device__ void TProlong(const SmemLevel<T> &F, const SmemLevel<T> &C)
{
    const int n = ListLen(F, 2);
    const T wv[2] = {(T)0.75, (T)0.25};
    for (int t = PhaseStart<kWarp>(); t < n; t += PhaseStride<kWarp>())
    {
        int a, b, d;
        Unpack(ListAt(F, 2, t), a, b, d);
        const int c = a * F.sI + b * F.sJ + d;
        const int A = (a + 1) >> 1, B = (b + 1) >> 1, D = k3D ? (d + 1) >> 1 : 0;
        const int si = (a & 1) ? -C.sI : C.sI, sj = (b & 1) ? -C.sJ : C.sJ, sk = (d & 1) ? -1 : 1;
        const int parent = A * C.sI + B * C.sJ + D;
        T acc = (T)0;
#pragma unroll
        for (int di = 0; di < 2; di++)
#pragma unroll
            for (int dj = 0; dj < 2; dj++)
#pragma unroll
                for (int dk = 0; dk < (k3D ? 2 : 1); dk++)
                {
                    // e is zero at SOLID (and all other non-unknown) contributors
                    const T w = wv[di] * wv[dj] * (k3D ? wv[dk] : (T)1);
                    acc += w * C.e[parent + di * si + dj * sj + dk * sk];
                }
        F.e[c] += acc + Moved(F, c) * C.e[parent];
    }
    PhaseSync<kWarp>();
}

// The descent through level l: the sweeps from zero, the residual and its restriction.
template <typename T, bool k3D, bool kSt, bool kWarp>
__device__ void TDown(const SmemLevel<T> &F, const SmemLevel<T> &C, int pre)
{
    TSweeps<T, k3D, kSt, kWarp>(F, pre, 0, true, true);
    TRestrict<T, k3D, kWarp>(F, C);
}

// The ascent into level l: the prolonged correction, then the post-sweeps black first.
template <typename T, bool k3D, bool kSt, bool kWarp>
__device__ void TUp(const SmemLevel<T> &F, const SmemLevel<T> &C, int post)
{
    TProlong<T, k3D, kWarp>(F, C);
    TSweeps<T, k3D, kSt, kWarp>(F, 0, post, false, false);
}

struct TailShared
{
    double inv[kMaxTailLevels][32]; // 1 / (gamma/2 * units), entry 0 = 0
    int count[kMaxTailLevels][2];
};

// What a layout fixes, into shared memory, and zeroed vectors: nothing here depends on the launch before.
template <typename T>
__device__ __forceinline__ void TailStage(const TailArgs<T> &A, unsigned char *smem, TailShared &sh)
{
    for (int t = threadIdx.x; t < 32 * A.nlev; t += blockDim.x)
    {
        const int l = t >> 5, u = t & 31;
        sh.inv[l][u] = u ? 1.0 / (0.5 * A.lv[l].v.gamma * (double)u) : 0.0;
        if (u < 2) sh.count[l][u] = A.counts[2 * l + u];
    }
    for (int l = 0; l < A.nlev; l++)
    {
        const SmemLevel<T> S = Bind<T>(A.lv[l], smem);
        const unsigned a = Pad16((unsigned)(S.cells * sizeof(T)));
        uint4 *z = reinterpret_cast<uint4 *>(S.r), *p = reinterpret_cast<uint4 *>(S.list);
        const uint4 *g = reinterpret_cast<const uint4 *>(A.lists + A.lv[l].listOff);
        for (unsigned t = threadIdx.x; t < A.lv[l].vecs * a / 16; t += blockDim.x) z[t] = make_uint4(0, 0, 0, 0);
        for (unsigned t = threadIdx.x; t < PrepBytes(S.cells) / 16; t += blockDim.x) p[t] = g[t];
    }
}

template <typename T, bool k3D, bool kSt>
__device__ __forceinline__ void TailBody(const TailArgs<T> &A, unsigned char *smem, const TailShared &sh)
{
    __syncthreads(); // the staged data; r of the first level overwrites its zeros
    {
        const SmemLevel<T> F0 = Bind<T>(A.lv[0], smem);
        for (int c = threadIdx.x; c < F0.cells; c += blockDim.x) F0.r[c] = A.rIn[c];
    }
    __syncthreads();
    auto lev = [&](int l) {
        SmemLevel<T> s = Bind<T>(A.lv[l], smem);
        s.nRed = sh.count[l][0];
        s.nBlack = sh.count[l][1];
        s.inv = sh.inv[l];
        return s;
    };
    const int last = A.nlev - 1;
    // wl: the first level from which every coarser one has at most 32 unknowns of each colour (warp 0 runs those)
    int wl = A.nlev;
    for (int l = last; l >= 0 && sh.count[l][0] <= 32 && sh.count[l][1] <= 32; l--) wl = l;
    const int top = wl < last ? wl : last;
    for (int l = 0; l < top; l++) TDown<T, k3D, kSt, false>(lev(l), lev(l + 1), A.pre);
    // the coarsest level: symmetric sweep pairs from zero
    if (wl > last) TSweeps<T, k3D, kSt, false>(lev(last), A.coarseSweeps, A.coarseSweeps, true, false);
    else
    {
        if (threadIdx.x < 32)
        {
            for (int l = wl; l < last; l++) TDown<T, k3D, kSt, true>(lev(l), lev(l + 1), A.pre);
            TSweeps<T, k3D, kSt, true>(lev(last), A.coarseSweeps, A.coarseSweeps, true, false);
            for (int l = last - 1; l >= wl; l--) TUp<T, k3D, kSt, true>(lev(l), lev(l + 1), A.post);
        }
        __syncthreads();
    }
    for (int l = top - 1; l >= 0; l--) TUp<T, k3D, kSt, false>(lev(l), lev(l + 1), A.post);
    const SmemLevel<T> F0 = Bind<T>(A.lv[0], smem);
    for (int c = threadIdx.x; c < F0.cells; c += blockDim.x) A.eOut[c] = F0.e[c];
}

template <typename T, bool k3D, bool kSt>
__global__ void __launch_bounds__(kTailThreadsBig, 1) k_tail(const __grid_constant__ TailArgs<T> A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TailShared sh;
    TailStage<T>(A, smem, sh); // written when the layout was set: before any launch this one may overlap
    PdlWait();
    PdlTrigger();
    TailBody<T, k3D, kSt>(A, smem, sh);
}

// batched (nb_batch.cu): block z runs the coarse end of the request at list[z], its arguments copied from global
// memory into shared memory first
__global__ void __launch_bounds__(kTailThreadsBig) kb_tail(const BatchReq *__restrict__ rq, BatchList a)
{
    extern __shared__ __align__(16) unsigned char smem[];
    PdlWait();
    PdlTrigger();
    const int q = BatchReqOf(a);
    if (q < 0) return;
    __shared__ TailArgs<float> sA;
    const TailArgs<float> *g = static_cast<const TailArgs<float> *>(rq[q].tail);
    {
        const int n = (int)(sizeof(TailArgs<float>) / sizeof(int));
        const int *src = reinterpret_cast<const int *>(g);
        int *dst = reinterpret_cast<int *>(&sA);
        for (int t = threadIdx.x; t < n; t += blockDim.x) dst[t] = src[t];
    }
    __syncthreads();
    __shared__ TailShared sh;
    TailStage<float>(sA, smem, sh);
    TailBody<float, true, false>(sA, smem, sh); // batches are uniform 3D
}

// Every tail level's prepared data, once per layout; the lists' order within a colour does not matter (the cells of one
// colour are updated independently).
__global__ void __launch_bounds__(1024) k_tail_lists(TailArgs<float> A)
{
    __shared__ int cnt[kMaxTailLevels][2];
    if (threadIdx.x < 2 * kMaxTailLevels) cnt[threadIdx.x >> 1][threadIdx.x & 1] = 0;
    __syncthreads();
    for (int l = 0; l < A.nlev; l++)
    {
        const LevelView &g = A.lv[l].v;
        const int cells = (int)g.cells, nq = g.dim == 3 ? 6 : 4;
        unsigned *list = const_cast<unsigned *>(A.lists) + A.lv[l].listOff;
        uint8_t *unit = (uint8_t *)list + Pad16((unsigned)cells * 4u), *ext = unit + Pad16((unsigned)cells);
        uint8_t *types = ext + Pad16((unsigned)cells);
        for (int c = threadIdx.x; c < cells; c += blockDim.x)
        {
            const unsigned code = g.code[c];
            unit[c] = g.stretched ? (uint8_t)code : (uint8_t)0;
            ext[c] = 0;
            types[c] = g.stretched ? g.types[c] : (uint8_t)0;
            if (!(code & CODE_UNKNOWN)) continue;
            const int k = c % g.Nz, rr = c / g.Nz, j = rr % g.Nx, i = rr / g.Nx;
            const int col = (i + j + k) & 1;
            const int pos = atomicAdd(&cnt[l][col], 1);
            const unsigned packed = ((unsigned)i << 20) | ((unsigned)j << 10) | (unsigned)k;
            if (col == 0) list[pos] = packed;
            else list[cells - 1 - pos] = packed;
            if (!g.stretched)
            {
                // half-units of the diagonal: 2 per FLUID neighbour, 2 per interior Dirichlet neighbour, 4 per
                // Dirichlet ring neighbour (ring factor 2)
                unsigned units = 2u * (unsigned)__popc(code & CODE_FLUID_MASK);
                if (code & CODE_DIRICHLET)
                    for (int q = 0; q < nq; q++)
                        if (IsDirichlet(g.types[c + NbrOffset(g, q)]))
                        {
                            const int ni = i + (q == 0) - (q == 1), nj = j + (q == 2) - (q == 3),
                                      nk = k + (q == 4) - (q == 5);
                            units += OnRing(g, ni, nj, nk) ? 4u : 2u;
                        }
                unit[c] = (uint8_t)(0x80u | units);
            }
            if (l + 1 < A.nlev)
            {
                // the trilinear (2D: bilinear) weights of the SOLID contributors, in 64ths
                const LevelView &cv = A.lv[l + 1].v;
                const bool d3 = g.dim == 3;
                const int si = (i & 1) ? -1 : 1, sj = (j & 1) ? -1 : 1, sk = (k & 1) ? -1 : 1;
                const long long parent = (long long)((i + 1) >> 1) * cv.sI + (long long)((j + 1) >> 1) * cv.sJ +
                                         (d3 ? (k + 1) >> 1 : 0);
                unsigned extra = 0;
                for (int q = 1; q < (d3 ? 8 : 4); q++)
                {
                    const int di = q & 1, dj = (q >> 1) & 1, dk = q >> 2;
                    if (cv.types[parent + (long long)(di * si) * cv.sI + (long long)(dj * sj) * cv.sJ + dk * sk] == SOLID)
                        extra += (di ? 1u : 3u) * (dj ? 1u : 3u) * (d3 ? (dk ? 1u : 3u) : 4u);
                }
                ext[c] = (uint8_t)(0x80u | extra);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 2 * A.nlev) const_cast<int *>(A.counts)[threadIdx.x] = cnt[threadIdx.x >> 1][threadIdx.x & 1];
}

long long TailListEntries(const LevelView *levels, int nlev)
{
    long long n = 0;
    for (int l = 0; l < nlev; l++) n += PrepBytes(levels[l].cells) / 4;
    return n;
}

// the levels' places in shared memory and in the prepared data; returns the shared memory's bytes
template <typename T> static unsigned PlaceLevels(TailArgs<T> &A, const LevelView *levels, int nlev)
{
    unsigned off = 0, listOff = 0;
    for (int l = 0; l < nlev; l++)
    {
        A.lv[l].v = levels[l];
        A.lv[l].off = off;
        A.lv[l].listOff = listOff;
        A.lv[l].vecs = l + 1 < nlev ? 3 : 2;
        off += LevelBytes<T>(levels[l].cells, l + 1 == nlev);
        listOff += PrepBytes(levels[l].cells) / 4;
    }
    A.nlev = nlev;
    return off;
}

void LaunchTailLists(const LevelView *levels, int nlev, unsigned *lists, int *counts, cudaStream_t st)
{
    TailArgs<float> A{};
    PlaceLevels(A, levels, nlev);
    A.lists = lists;
    A.counts = counts;
    NB_COUNT_LAUNCH();
    k_tail_lists<<<1, 1024, 0, st>>>(A);
}

template <typename T> size_t TailSmemBytes(const LevelView *levels, int nlev)
{
    size_t bytes = 0;
    for (int l = 0; l < nlev; l++) bytes += LevelBytes<T>(levels[l].cells, l + 1 == nlev);
    return bytes;
}

template <typename T> static bool PrepareTailOnce()
{
    auto ok = [](const void *f) {
        return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailMaxSmem) == cudaSuccess;
    };
    if (sizeof(T) == 4 && !ok((const void *)kb_tail)) return false;
    return ok((const void *)k_tail<T, false, false>) && ok((const void *)k_tail<T, false, true>) &&
           ok((const void *)k_tail<T, true, false>) && ok((const void *)k_tail<T, true, true>);
}

// Once per device and precision: changing a kernel's attribute on every layout change would take the driver's
// locks under a server's running solves.
template <typename T> bool PrepareTail(size_t bytes)
{
    if (bytes > kTailMaxSmem) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    static std::mutex mu;
    static std::set<int> done;
    std::lock_guard<std::mutex> lock(mu);
    const int key = 2 * dev + (sizeof(T) == 4 ? 0 : 1);
    if (done.count(key)) return true;
    if (!PrepareTailOnce<T>()) return false;
    done.insert(key);
    return true;
}
// The coarse end's arguments of one request (FP32), for a batch's table in device memory: *bytes = their size,
// and when out is not null they are written there; *smem = the dynamic shared memory of its launch.
void TailArgsFor(const LevelView *levels, int nlev, const float *rIn, float *eOut, int pre, int post,
                 int coarseSweeps, const unsigned *lists, const int *counts, void *out, size_t *bytes, size_t *smem)
{
    TailArgs<float> A{};
    const unsigned off = PlaceLevels(A, levels, nlev);
    A.rIn = rIn;
    A.eOut = eOut;
    A.pre = pre < 1 ? 1 : pre;
    A.post = post < 1 ? 1 : post;
    A.coarseSweeps = coarseSweeps < 1 ? 1 : coarseSweeps;
    A.lists = lists;
    A.counts = counts;
    *bytes = sizeof(A);
    *smem = off;
    if (out) std::memcpy(out, &A, sizeof(A));
}

void LaunchBatchTail(const BatchReq *rq, BatchList a, int cap, size_t smem, cudaStream_t st)
{
    NB_COUNT_LAUNCH();
    LaunchPdl(kb_tail, dim3(1, 1, cap), dim3(kTailThreads), smem, st, rq, a);
}

template <typename T>
void LaunchTail(const LevelView *levels, int nlev, const T *rIn, T *eOut, int pre, int post, int coarseSweeps,
                const unsigned *lists, const int *counts, cudaStream_t st)
{
    TailArgs<T> A{};
    const unsigned off = PlaceLevels(A, levels, nlev);
    A.rIn = rIn;
    A.eOut = eOut;
    A.pre = pre < 1 ? 1 : pre;
    A.post = post < 1 ? 1 : post;
    A.coarseSweeps = coarseSweeps < 1 ? 1 : coarseSweeps;
    A.lists = lists;
    A.counts = counts;
    const dim3 threads(levels[0].cells > 4 * kTailThreads ? kTailThreadsBig : kTailThreads);
    NB_COUNT_LAUNCH();
    if (levels[0].dim == 3 && !levels[0].stretched)
        LaunchPdl(k_tail<T, true, false>, dim3(1), threads, (size_t)off, st, A);
    else if (levels[0].dim == 3)
        LaunchPdl(k_tail<T, true, true>, dim3(1), threads, (size_t)off, st, A);
    else if (!levels[0].stretched)
        LaunchPdl(k_tail<T, false, false>, dim3(1), threads, (size_t)off, st, A);
    else
        LaunchPdl(k_tail<T, false, true>, dim3(1), threads, (size_t)off, st, A);
}

template size_t TailSmemBytes<float>(const LevelView *, int);
template size_t TailSmemBytes<double>(const LevelView *, int);
template bool PrepareTail<float>(size_t);
template bool PrepareTail<double>(size_t);
template void LaunchTail<float>(const LevelView *, int, const float *, float *, int, int, int, const unsigned *,
                                const int *, cudaStream_t);
template void LaunchTail<double>(const LevelView *, int, const double *, double *, int, int, int, const unsigned *,
                                 const int *, cudaStream_t);

} // namespace nb
