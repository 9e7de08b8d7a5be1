// Building blocks of the colour-split kernels (nb_split.cu, nb_stretched.cu): 16-byte quads of one colour, a thread's
// position and march, idle tiles, launch grids.
#pragma once

#include "nb_kernels.h"

namespace nb
{

namespace
{

// the 16 bytes a thread moves at a time
template <typename T> struct Quad
{
    static constexpr int N = 16 / (int)sizeof(T);
    T v[N];
};
template <typename T> constexpr int kQ = Quad<T>::N;

__device__ __forceinline__ Quad<float> LQ(const float *p)
{
    const float4 a = *reinterpret_cast<const float4 *>(p);
    return Quad<float>{{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ Quad<double> LQ(const double *p)
{
    const double2 a = *reinterpret_cast<const double2 *>(p);
    return Quad<double>{{a.x, a.y}};
}
__device__ __forceinline__ void SQ(float *p, const Quad<float> &a)
{
    *reinterpret_cast<float4 *>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
__device__ __forceinline__ void SQ(double *p, const Quad<double> &a)
{
    *reinterpret_cast<double2 *>(p) = make_double2(a.v[0], a.v[1]);
}
// loads of values a kernel reads once (evict-first): measured to keep the half-sweep's j-row loads in L1 longer
__device__ __forceinline__ Quad<float> LQOnce(const float *p)
{
    const float4 a = __ldcs(reinterpret_cast<const float4 *>(p));
    return Quad<float>{{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ Quad<double> LQOnce(const double *p)
{
    const double2 a = __ldcs(reinterpret_cast<const double2 *>(p));
    return Quad<double>{{a.x, a.y}};
}
// a quad's N bytes of a byte array
template <int N> __device__ __forceinline__ unsigned LdB(const uint8_t *p)
{
    static_assert(N == 4 || N == 2, "four or two bytes");
    if constexpr (N == 4) return *reinterpret_cast<const unsigned *>(p);
    else return *reinterpret_cast<const unsigned short *>(p);
}
template <int N> __device__ __forceinline__ unsigned LdBOnce(const uint8_t *p)
{
    if constexpr (N == 4) return __ldcs(reinterpret_cast<const unsigned *>(p));
    else return __ldcs(reinterpret_cast<const unsigned short *>(p));
}
__device__ __forceinline__ unsigned Byte(unsigned d, int x) { return (d >> (8 * x)) & 0xFFu; }
template <typename T> __device__ __forceinline__ T Unk(unsigned b) { return (b & 0x80u) ? (T)1 : (T)0; }

// 1 / (gamma/2 * units), entry 0 = 0
template <typename T> __device__ __forceinline__ void FillInv(T *inv, double gamma)
{
    if (threadIdx.x < 32) inv[threadIdx.x] = threadIdx.x ? (T)1 / ((T)0.5 * (T)gamma * (T)threadIdx.x) : (T)0;
    __syncthreads();
}

// Per-thread position of a quad kernel.
struct QuadPos
{
    int lane;
    bool valid;  // false for the clamped threads past the plane's last quad (they still load and shuffle)
    int i0, i1;  // planes [i0, i1)
    int j, m0;   // row and first element of the quad
    int RS, PS;
    long long off; // element of the quad on plane i0, within one colour
};

template <int N> __device__ __forceinline__ QuadPos QuadStart(const LevelView &v, const Blk &b)
{
    QuadPos p;
    const int Q = v.sRS / N, nq = v.Nx * Q;
    p.lane = threadIdx.x & 31;
    int t = b.x * kPairThreads + threadIdx.x;
    p.valid = t < nq;
    if (!p.valid) t = nq - 1;
    // grid.y splits the Ny-2 interior planes into chunks of S (the host sized it); a block past the last plane starts
    // at the ring plane and marches none
    const int S = (v.Ny - 2 + b.gy - 1) / b.gy;
    p.i0 = min(1 + b.y * S, v.Ny - 1);
    p.i1 = min(p.i0 + S, v.Ny - 1);
    p.RS = v.sRS;
    p.PS = v.sPS;
    p.j = t / Q;
    p.m0 = N * (t - p.j * Q);
    p.off = (long long)p.i0 * v.sPS + (long long)N * t;
    return p;
}

// True when no tile this block owns on planes [i0, i1) holds an unknown (LevelView::act): the block's cells are
// all zero in every vector and stay so, so it has nothing to compute, load or store.
__device__ __forceinline__ bool TileIdle(const LevelView &v, int bx, int i0, int i1)
{
    if (!v.act) return false;
    for (int i = i0; i < i1; i++)
        if (v.act[(long long)i * v.actTiles + bx]) return false;
    return true;
}

// The same for a block of a grid-layout pair kernel (PairStart): its rows j0 .. j1 of planes [i0, i1), checked
// through the split tiles (of kTile elements) that hold those rows' cells in either colour.
template <int kTile> __device__ __forceinline__ bool RowsIdle(const LevelView &v, int j0, int j1, int i0, int i1)
{
    if (!v.act) return false;
    const int t0 = (int)(((long long)j0 * v.sRS) / kTile);
    const int t1 = min(v.actTiles - 1, (int)(((long long)(j1 + 1) * v.sRS - 1) / kTile));
    for (int i = i0; i < i1; i++)
        for (int t = t0; t <= t1; t++)
            if (v.act[(long long)i * v.actTiles + t]) return false;
    return true;
}

// Resident blocks of a kernel per SM at kPairThreads threads (its registers and shared memory decide), and the SM
// count of the current device.
inline int ResidentBlocks(const void *fn)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kPairThreads, 0) != cudaSuccess || n < 1) n = 1;
    return n;
}

// read once per kernel (and before any stream capture: PrepareSplitKernels)
template <auto kKernel> int Occ()
{
    static const int n = ResidentBlocks((const void *)kKernel);
    return n;
}

inline int SmCount()
{
    int d = 0, c = 0;
    if (cudaGetDevice(&d) != cudaSuccess) return 148;
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || c < 1) c = 148;
    return c;
}

// The launch grid of a quad kernel with `resident` blocks per SM: the longest march (planes per thread, at most
// kQuadMaxS) whose launch fills the last wave of resident blocks to at least 90%; the longer the march, the fewer
// planes of a neighbour array are loaded twice (a chunk of S planes loads S + 2). Measured on a 258^3 level: one
// 92%-full wave of 16-plane chunks beats two waves of 8 (and 1.03 waves of 15 runs at half speed). With no such S,
// the best-filled one (a small level fills no wave: S = 1, all the parallelism there is).
constexpr int kQuadMaxS = 16;

// The march length S (planes per thread, 1 .. kQuadMaxS) for a grid of perPlane x ceil(planes / S) blocks on `slots`
// resident blocks, by the rule above.
inline long long BestMarch(long long perPlane, long long planes, long long slots)
{
    long long bestS = 1;
    double bestU = -1.0;
    for (long long S = kQuadMaxS; S >= 1; S--)
    {
        const long long blocks = perPlane * ((planes + S - 1) / S);
        const long long waves = (blocks + slots - 1) / slots;
        const double u = (double)blocks / (double)(waves * slots);
        if (u >= 0.9) return S;
        if (u > bestU + 1e-9)
        {
            bestU = u;
            bestS = S;
        }
    }
    return bestS;
}

// A quad kernel's grid with a march of S planes (S > 0), or sized as above (S = 0); N elements a thread.
template <int N = 4> inline dim3 QuadGridS(const LevelView &v, int S)
{
    const long long nq = (long long)v.Nx * (v.sRS / N), perPlane = (nq + kPairThreads - 1) / kPairThreads;
    const long long planes = v.Ny - 2 > 0 ? v.Ny - 2 : 1;
    return dim3((unsigned)perPlane, (unsigned)((planes + S - 1) / S));
}

template <int N> inline dim3 QuadGrid(const LevelView &v, int resident)
{
    const long long nq = (long long)v.Nx * (v.sRS / N), perPlane = (nq + kPairThreads - 1) / kPairThreads;
    const long long planes = v.Ny - 2 > 0 ? v.Ny - 2 : 1;
    const long long bestS = BestMarch(perPlane, planes, (long long)SmCount() * (resident > 0 ? resident : 1));
    return dim3((unsigned)perPlane, (unsigned)((planes + bestS - 1) / bestS));
}

// The other colour's k neighbours of a quad: the element at m (c) and the one at m + (q ? 1 : -1) (returned).
__device__ __forceinline__ Quad<float> KShift(const Quad<float> &c, float prevW, float nextX, int q)
{
    return q ? Quad<float>{{c.v[1], c.v[2], c.v[3], nextX}} : Quad<float>{{prevW, c.v[0], c.v[1], c.v[2]}};
}
__device__ __forceinline__ Quad<double> KShift(const Quad<double> &c, double prevW, double nextX, int q)
{
    return q ? Quad<double>{{c.v[1], nextX}} : Quad<double>{{prevW, c.v[0]}};
}

// The elements just before and after this lane's quad in its row (0 past the row's ends; the values a lane takes
// from a neighbouring row only reach ring or padding cells, whose results are masked).
template <typename T>
__device__ __forceinline__ void Edges(const QuadPos &P, const Quad<T> &c, const T *row, T &prevW, T &nextX)
{
    constexpr int N = kQ<T>;
    prevW = __shfl_up_sync(0xffffffffu, c.v[N - 1], 1);
    nextX = __shfl_down_sync(0xffffffffu, c.v[0], 1);
    if (P.lane == 0) prevW = P.m0 > 0 ? row[-1] : (T)0;
    if (P.lane == 31) nextX = P.m0 + N < P.RS ? row[N] : (T)0;
}

} // namespace

} // namespace nb
