// Boundary-condition replay on the device: MAC::EnforceVelocityBC and MAC::EnforcePressureBC (src/MAC.cpp:811-865)
// from the lists MAC::BuildBoundaryLists makes on the host (src/MAC.cpp:613-1090), so that a stepping loop can keep
// u, v, w and p on the device between its sub-steps. The fields come out bit for bit as the reference's serial
// replay leaves them.
//
// The reference replays, in order: zeros on solidFaceList[c]; the boundary velocity function's values on
// prescribedList (when the scene has one); copies f[dst] = f[src] on copyList (a corner copies from an edge that
// copied from a face, so the order matters); ApplyOutflowFlux; and, for p, ringList (zero, prescribed value or copy).
// Here the writes of one call form a program of (field, dst, source) operations, grouped once, at creation, into
// levels: an operation goes one level after the last earlier write of its destination, after every earlier read of
// its destination, and after the last earlier write of its source. Operations of one level touch distinct
// destinations and read nothing another operation of the level writes, so each level is one race-free scatter launch
// and the levels in turn give exactly the sequential result. Leaving out the prescribed writes (no velocity
// function) keeps that true: a removed write only ever added ordering.
//
// Most programs need no levels at all (LevelProgram's flat form): what a destination holds at the end is zero, one of the
// values, or what some entry held before the call, found at creation by following its last write's copies back. Where
// no such entry is itself written, the resolved writes are independent and the replay is one launch. Consecutive ones
// that step by constant strides (a face of the grid, a row) become runs, so that a warp reads 32 bytes of program for
// up to 256 writes instead of 16 for each. A channel of 256^3 with an inlet, an outlet and a solid sphere, both replays
// (B200): 45-47 us as five levels of single operations, 34.7 us as two launches of runs.
//
// ApplyOutflowFlux sums sign * f * area over the inlet and the outflow faces in list order; one block forms the
// products in parallel, one thread adds them in the reference's order (so the correction rounds as the reference's
// does), and the block applies it. The prescribed values (the tinyexpr boundary functions) are evaluated by the
// caller on the host, as the reference does, and passed per call as a device array in list order.
#include "nb_solver.h"

#include <algorithm>
#include <cstdint>
#include <memory>
#include <vector>

namespace nb
{

namespace
{

constexpr int kBcThreads = 256;
constexpr int kFluxThreads = 512;

struct BcOp
{
    int32_t comp; // field: 0 u, 1 v, 2 w (velocity); 0 p (pressure)
    int32_t dst;
    int32_t src;  // >= 0: copy f[src]
    int32_t val;  // src < 0, val >= 0: values[val]; both < 0: zero
};

__global__ void __launch_bounds__(kBcThreads)
    k_bc_level(const BcOp *__restrict__ ops, int n, double *f0, double *f1, double *f2,
               const double *__restrict__ values, int nullValuesZero)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
    {
        const BcOp o = ops[q];
        double *f = o.comp == 0 ? f0 : (o.comp == 1 ? f1 : f2);
        if (o.src >= 0)
            f[o.dst] = f[o.src];
        else if (o.val >= 0)
        {
            if (values) f[o.dst] = values[o.val];
            else if (nullValuesZero) f[o.dst] = 0.0;
        }
        else
            f[o.dst] = 0.0;
    }
}

// n writes f[dst + k dd] = f[src + k ds] (src >= 0), values[val + k dv] (val >= 0) or 0, k = 0 .. n-1
struct alignas(32) BcRun
{
    int32_t comp, n, dst, dd, src, ds, val, dv;
};
constexpr int kRunMax = 256; // writes of a run at most: eight a lane

// A resolved program: one warp per run. values null: the pressure replay's zeros (a velocity program without values
// holds no such run).
__global__ void __launch_bounds__(kBcThreads)
    k_bc_runs(const BcRun *__restrict__ runs, int n, double *f0, double *f1, double *f2,
              const double *__restrict__ values)
{
    const int lane = threadIdx.x & 31, q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (q >= n) return;
    const BcRun r = runs[q];
    double *f = r.comp == 0 ? f0 : (r.comp == 1 ? f1 : f2);
    double x[kRunMax / 32];
#pragma unroll
    for (int b = 0; b < kRunMax / 32; b++)
    {
        const int k = lane + 32 * b;
        x[b] = 0.0;
        if (k >= r.n) continue;
        if (r.src >= 0) x[b] = f[r.src + k * r.ds];
        else if (r.val >= 0 && values) x[b] = values[r.val + k * r.dv];
    }
#pragma unroll
    for (int b = 0; b < kRunMax / 32; b++)
        if (lane + 32 * b < r.n) f[r.dst + (lane + 32 * b) * r.dd] = x[b];
}

struct FluxFaces
{
    const int32_t *comp, *index, *outer; // inlet faces first (outer unused), then the outflow faces
    const double *area, *sign;
    int nin, nout;
    double aOut;                         // sum of the outflow areas, in list order (host)
};

__global__ void __launch_bounds__(kFluxThreads) k_bc_outflow(FluxFaces ff, double *f0, double *f1, double *f2,
                                                             double *prod)
{
    __shared__ double delta;
    const int n = ff.nin + ff.nout;
    for (int q = threadIdx.x; q < n; q += blockDim.x)
    {
        const double *f = ff.comp[q] == 0 ? f0 : (ff.comp[q] == 1 ? f1 : f2);
        prod[q] = ff.sign[q] * f[ff.index[q]] * ff.area[q];
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double qIn = 0.0, qOut = 0.0;
        for (int q = 0; q < ff.nin; q++) qIn -= prod[q];
        for (int q = ff.nin; q < n; q++) qOut += prod[q];
        delta = (qIn - qOut) / ff.aOut;
    }
    __syncthreads();
    for (int q = ff.nin + threadIdx.x; q < n; q += blockDim.x)
    {
        double *f = ff.comp[q] == 0 ? f0 : (ff.comp[q] == 1 ? f1 : f2);
        const double v = f[ff.index[q]] + ff.sign[q] * delta;
        f[ff.index[q]] = v;
        f[ff.outer[q]] = v;
    }
}

// Field entry -> int, open addressing (the programs hold a million entries and more: node-based maps took most of the
// plan's time)
class EntryMap
{
  public:
    explicit EntryMap(size_t entries)
    {
        size_t n = 16;
        while (n < entries + entries / 2) n *= 2;
        keys.assign(n, -1);
        vals.resize(n);
    }
    static long long Key(int comp, int index) { return ((long long)comp << 32) | (unsigned)index; }
    // the value of a key, or null
    int *Find(long long k)
    {
        const size_t at = Slot(k);
        return keys[at] == k ? &vals[at] : nullptr;
    }
    void Set(long long k, int v)
    {
        const size_t at = Slot(k);
        keys[at] = k;
        vals[at] = v;
    }

  private:
    std::vector<long long> keys;
    std::vector<int> vals;
    size_t Slot(long long k) const
    {
        const size_t mask = keys.size() - 1;
        // sixteen neighbouring entries stay together: faces are walked in order
        size_t at = ((size_t)(((unsigned long long)(k >> 4) * 0x9E3779B97F4A7C15ull) >> 24) * 16 + (size_t)(k & 15)) & mask;
        while (keys[at] != -1 && keys[at] != k) at = (at + 1) & mask;
        return at;
    }
};

// Levels of a sequential write program (see the top of this file): the operations sorted by level (stable), the start
// of each level and each operation's level in program order. flat (may be null): also the independent writes that
// leave what the sequence leaves, one per destination, its source traced back through the copies to zero, a value or
// an entry's content before the call; returns false (and leaves flat empty) when an entry read that way is also
// written, so that the order counts.
bool LevelProgram(const std::vector<BcOp> &seq, std::vector<BcOp> &sorted, std::vector<int> &start,
                  std::vector<int> &level, std::vector<BcOp> *flat)
{
    size_t copies = 0;
    for (const BcOp &o : seq) copies += o.src >= 0;
    EntryMap last(seq.size()), lastRead(copies); // an entry's last write (its number), last read (its level)
    std::vector<BcOp> res;
    if (flat) res = seq;
    level.assign(seq.size(), 0);
    int nlev = 0;
    for (size_t q = 0; q < seq.size(); q++)
    {
        const BcOp &o = seq[q];
        int l = 0;
        const long long kd = EntryMap::Key(o.comp, o.dst);
        if (const int *w = last.Find(kd)) l = level[*w] + 1;
        if (const int *v = lastRead.Find(kd)) l = std::max(l, *v + 1);
        if (o.src >= 0)
        {
            const long long ks = EntryMap::Key(o.comp, o.src);
            if (const int *w = last.Find(ks))
            {
                l = std::max(l, level[*w] + 1);
                if (flat)
                {
                    res[q].src = res[*w].src;
                    res[q].val = res[*w].val;
                }
            }
            const int *v = lastRead.Find(ks);
            if (!v || *v < l) lastRead.Set(ks, l);
        }
        last.Set(kd, (int)q);
        level[q] = l;
        if (l + 1 > nlev) nlev = l + 1;
    }
    start.assign(nlev + 1, 0);
    for (size_t q = 0; q < seq.size(); q++) start[level[q] + 1]++;
    for (int l = 0; l < nlev; l++) start[l + 1] += start[l];
    std::vector<int> fill(start.begin(), start.end() - 1);
    sorted.resize(seq.size());
    for (size_t q = 0; q < seq.size(); q++) sorted[fill[level[q]]++] = seq[q];
    if (!flat) return false;
    flat->clear();
    for (size_t q = 0; q < seq.size(); q++)
    {
        const BcOp &o = res[q];
        if (*last.Find(EntryMap::Key(o.comp, o.dst)) != (int)q || o.src == o.dst) continue; // overwritten, or as it was
        if (o.src >= 0)
        {
            const int *w = last.Find(EntryMap::Key(o.comp, o.src));
            if (w && res[*w].src != o.src)
            {
                flat->clear();
                return false;
            }
        }
        flat->push_back(o);
    }
    return true;
}

// Consecutive operations of constant strides as runs, appended to `runs`; those of fewer than `least` writes go to `rest`
// operation by operation instead.
void TakeRuns(const std::vector<BcOp> &ops, size_t least, std::vector<BcRun> &runs, std::vector<BcOp> &rest)
{
    auto kind = [](const BcOp &o) { return o.src >= 0 ? 0 : (o.val >= 0 ? 1 : 2); };
    for (size_t q = 0; q < ops.size();)
    {
        const BcOp &a = ops[q];
        BcRun r{a.comp, 1, a.dst, 0, a.src, 0, a.val, 0};
        auto joins = [&](const BcOp &b) {
            const long long k = r.n;
            return b.comp == a.comp && kind(b) == kind(a) && b.dst == r.dst + k * r.dd &&
                   (a.src < 0 || b.src == r.src + k * r.ds) && (a.src >= 0 || a.val < 0 || b.val == r.val + k * r.dv);
        };
        if (q + 1 < ops.size())
        {
            const BcOp &b = ops[q + 1];
            r.dd = b.dst - a.dst;
            r.ds = a.src >= 0 ? b.src - a.src : 0;
            r.dv = a.src < 0 && a.val >= 0 ? b.val - a.val : 0;
        }
        size_t e = q + 1;
        while (e < ops.size() && r.n < kRunMax && joins(ops[e])) r.n++, e++;
        if ((size_t)r.n < least) rest.insert(rest.end(), ops.begin() + q, ops.begin() + e);
        else
        {
            if (r.n == 1) r.dd = r.ds = r.dv = 0;
            runs.push_back(r);
        }
        q = e;
    }
}

// The operations as runs: those that follow each other in the list (rows, faces across the slow axes), then, of the
// rest, those in the same place of consecutive rows (the faces at both ends of the fast axis, whose entries alternate
// in the list). Empty when they come out too short for a warp each (fewer than eight writes a run on average).
// row[c]: entries of a row of field c.
void MakeRuns(const std::vector<BcOp> &ops, const int row[3], std::vector<BcRun> &runs)
{
    runs.clear();
    std::vector<BcOp> rest, byPlace;
    TakeRuns(ops, 8, runs, rest);
    if (!rest.empty())
    {
        // stable, by field and place in the row
        const int base[4] = {0, row[0], row[0] + row[1], row[0] + row[1] + row[2]};
        auto place = [&](const BcOp &o) { return base[o.comp] + o.dst % row[o.comp]; };
        std::vector<size_t> at((size_t)base[3] + 1, 0);
        for (const BcOp &o : rest) at[place(o) + 1]++;
        for (size_t p = 1; p < at.size(); p++) at[p] += at[p - 1];
        byPlace.resize(rest.size());
        for (const BcOp &o : rest) byPlace[at[place(o)]++] = o;
        rest.clear();
        TakeRuns(byPlace, 1, runs, rest);
    }
    if (runs.size() * 8 > ops.size()) runs.clear();
}

// A replay's resolved forms on the host, where it resolves (ok): runs, or single operations where runs is empty
struct Resolved
{
    bool ok = false;
    std::vector<BcOp> ops;
    std::vector<BcRun> runs;
};

} // namespace

// A resolved replay on the device
struct BcFlat
{
    bool ok = false;
    int nOps = 0, nRuns = 0;
    DevArray<BcOp> ops;
    DevArray<BcRun> runs;
    void Upload(const Resolved &r)
    {
        ok = r.ok;
        nRuns = (int)r.runs.size();
        nOps = nRuns ? 0 : (int)r.ops.size();
        if (nRuns) runs.upload(r.runs.data(), r.runs.size(), 0);
        if (nOps) ops.upload(r.ops.data(), r.ops.size(), 0);
    }
};

struct BcReplay
{
    int device = 0;
    int dim = 3;
    int npresc = 0, nring = 0;
    BcFlat velFlat, presFlat;
    DevArray<BcOp> vel, pres; // the levelled programs: replays that do not resolve, and velocities without values
    std::vector<int> velStart, presStart;
    DevArray<int32_t> fluxI;  // comp | index | outer, each nin + nout
    DevArray<double> fluxD;   // area | sign | products
    FluxFaces ff{};
};

struct BcHost
{
    int dim = 3, npresc = 0, nring = 0, nin = 0, nout = 0;
    std::vector<BcOp> vel, pres;
    Resolved velR, presR;
    std::vector<int> velStart, presStart;
    std::vector<int> velLevel, presLevel; // each operation's level, in list order
    std::vector<int32_t> fluxI;
    std::vector<double> fluxD;
    double aOut = 0.0;
};

namespace
{
void CheckIndex(long long i, long long size, const char *what)
{
    if (i < 0 || i >= size) throw InputError(std::string(what) + " index outside its field");
}
} // namespace

// resolve: also the resolved programs (a replay that runs needs them, the plan of the levels does not)
static BcHost BuildBcHost(const nb_bc_lists &L, bool resolve)
{
    if (L.dim != 2 && L.dim != 3) throw InputError("dim must be 2 or 3");
    const long long nz = L.dim == 3 ? L.Nz : 1;
    if (L.Nx < 1 || L.Ny < 1 || nz < 1) throw InputError("bad sizes");
    const long long Nx = L.Nx, Ny = L.Ny;
    const long long sizes[3] = {(Nx + 1) * Ny * nz, Nx * (Ny + 1) * nz, L.dim == 3 ? Nx * Ny * (nz + 1) : 0};
    const long long pSize = Nx * Ny * nz;
    for (long long s : sizes)
        if (s >= (1ll << 31)) throw InputError("fields of at most 2^31 - 1 entries");
    auto counts_ok = [](int n, const void *p) { return n == 0 || (n > 0 && p); };
    for (int c = 0; c < 3; c++)
        if (!counts_ok(L.nsolid[c], L.solid[c])) throw InputError("solid face list");
    if (!counts_ok(L.npresc, L.presc_comp) || !counts_ok(L.npresc, L.presc_index)) throw InputError("prescribed list");
    if (!counts_ok(L.ncopy, L.copy_comp) || !counts_ok(L.ncopy, L.copy_dst) || !counts_ok(L.ncopy, L.copy_src))
        throw InputError("copy list");
    if (!counts_ok(L.nring, L.ring_dst) || !counts_ok(L.nring, L.ring_kind) || !counts_ok(L.nring, L.ring_src))
        throw InputError("ring list");
    if (!counts_ok(L.ninlet, L.inlet_comp) || !counts_ok(L.ninlet, L.inlet_index) ||
        !counts_ok(L.ninlet, L.inlet_area) || !counts_ok(L.ninlet, L.inlet_sign))
        throw InputError("inlet faces");
    if (!counts_ok(L.noutflow, L.outflow_comp) || !counts_ok(L.noutflow, L.outflow_index) ||
        !counts_ok(L.noutflow, L.outflow_outer) || !counts_ok(L.noutflow, L.outflow_area) ||
        !counts_ok(L.noutflow, L.outflow_sign))
        throw InputError("outflow faces");
    const int ncomp = L.dim == 3 ? 3 : 2;
    auto comp_ok = [&](int c) {
        if (c < 0 || c >= ncomp) throw InputError("velocity component out of range");
        return c;
    };

    std::vector<BcOp> seq;
    seq.reserve((size_t)L.nsolid[0] + L.nsolid[1] + L.nsolid[2] + L.npresc + L.ncopy);
    for (int c = 0; c < 3; c++)
        for (int q = 0; q < L.nsolid[c]; q++)
        {
            comp_ok(c);
            CheckIndex(L.solid[c][q], sizes[c], "solid face");
            seq.push_back({c, L.solid[c][q], -1, -1});
        }
    for (int q = 0; q < L.npresc; q++)
    {
        const int c = comp_ok(L.presc_comp[q]);
        CheckIndex(L.presc_index[q], sizes[c], "prescribed");
        seq.push_back({c, L.presc_index[q], -1, q});
    }
    for (int q = 0; q < L.ncopy; q++)
    {
        const int c = comp_ok(L.copy_comp[q]);
        CheckIndex(L.copy_dst[q], sizes[c], "copy destination");
        CheckIndex(L.copy_src[q], sizes[c], "copy source");
        seq.push_back({c, L.copy_dst[q], L.copy_src[q], -1});
    }
    std::vector<BcOp> pseq;
    pseq.reserve(L.nring);
    for (int q = 0; q < L.nring; q++)
    {
        CheckIndex(L.ring_dst[q], pSize, "ring destination");
        const int kind = L.ring_kind[q];
        if (kind < 0 || kind > 2) throw InputError("ring kind must be 0, 1 or 2");
        if (kind == 2) CheckIndex(L.ring_src[q], pSize, "ring source");
        pseq.push_back({0, L.ring_dst[q], kind == 2 ? L.ring_src[q] : -1, kind == 1 ? q : -1});
    }
    const int nin = L.ninlet, nout = L.noutflow;
    std::vector<int32_t> fi(3 * (size_t)(nin + nout), 0);
    std::vector<double> fd(3 * (size_t)(nin + nout), 0.0);
    double aOut = 0.0;
    for (int q = 0; q < nin + nout; q++)
    {
        const bool out = q >= nin;
        const int r = out ? q - nin : q;
        const int c = comp_ok(out ? L.outflow_comp[r] : L.inlet_comp[r]);
        const int idx = out ? L.outflow_index[r] : L.inlet_index[r];
        CheckIndex(idx, sizes[c], "flux face");
        fi[q] = c;
        fi[(nin + nout) + q] = idx;
        if (out)
        {
            CheckIndex(L.outflow_outer[r], sizes[c], "flux face outer");
            fi[2 * (nin + nout) + q] = L.outflow_outer[r];
            aOut += L.outflow_area[r];
        }
        fd[q] = out ? L.outflow_area[r] : L.inlet_area[r];
        fd[(nin + nout) + q] = out ? L.outflow_sign[r] : L.inlet_sign[r];
    }

    BcHost h;
    h.dim = L.dim;
    h.npresc = L.npresc;
    h.nring = L.nring;
    h.velR.ok = LevelProgram(seq, h.vel, h.velStart, h.velLevel, resolve ? &h.velR.ops : nullptr);
    h.presR.ok = LevelProgram(pseq, h.pres, h.presStart, h.presLevel, resolve ? &h.presR.ops : nullptr);
    const int fast = (int)(L.dim == 3 ? nz : Nx);
    const int rowV[3] = {L.dim == 3 ? fast : fast + 1, fast, L.dim == 3 ? fast + 1 : 1}, rowP[3] = {fast, 1, 1};
    MakeRuns(h.velR.ops, rowV, h.velR.runs);
    MakeRuns(h.presR.ops, rowP, h.presR.runs);
    h.fluxI.swap(fi);
    h.fluxD.swap(fd);
    h.nin = nin;
    h.nout = nout;
    h.aOut = aOut;
    return h;
}

static BcReplay *CreateBcReplay(int device, const BcHost &h)
{
    std::unique_ptr<BcReplay> b(new BcReplay);
    b->device = device;
    b->dim = h.dim;
    b->npresc = h.npresc;
    b->nring = h.nring;
    b->velStart = h.velStart;
    b->presStart = h.presStart;
    b->velFlat.Upload(h.velR);
    b->presFlat.Upload(h.presR);
    if ((!h.velR.ok || h.npresc > 0) && !h.vel.empty()) b->vel.upload(h.vel.data(), h.vel.size(), 0);
    if (!h.presR.ok && !h.pres.empty()) b->pres.upload(h.pres.data(), h.pres.size(), 0);
    const int n = h.nin + h.nout;
    if (n > 0)
    {
        b->fluxI.upload(h.fluxI.data(), h.fluxI.size(), 0);
        b->fluxD.upload(h.fluxD.data(), h.fluxD.size(), 0);
    }
    NB_CK(cudaStreamSynchronize(0));
    b->ff.comp = b->fluxI.p;
    b->ff.index = b->fluxI.p ? b->fluxI.p + n : nullptr;
    b->ff.outer = b->fluxI.p ? b->fluxI.p + 2 * n : nullptr;
    b->ff.area = b->fluxD.p;
    b->ff.sign = b->fluxD.p ? b->fluxD.p + n : nullptr;
    b->ff.nin = h.nin;
    b->ff.nout = h.nout;
    b->ff.aOut = h.aOut;
    return b.release();
}

void CheckBcLists(const nb_bc_lists &lists) { (void)BuildBcHost(lists, false); }

void PlanBcLevels(const nb_bc_lists &lists, std::vector<int> &velocity, std::vector<int> &pressure)
{
    BcHost h = BuildBcHost(lists, false);
    velocity.swap(h.velLevel);
    pressure.swap(h.presLevel);
}

BcReplay *CreateBcReplay(int device, const nb_bc_lists &lists) { return CreateBcReplay(device, BuildBcHost(lists, true)); }

void DestroyBcReplay(BcReplay *b) { delete b; }

int BcLevels(const BcReplay &b, int pressure) { return (int)(pressure ? b.presStart : b.velStart).size() - 1; }

int BcDevice(const BcReplay &b) { return b.device; }

namespace
{
void RunLevels(const DevArray<BcOp> &ops, const std::vector<int> &start, double *f0, double *f1, double *f2,
               const double *values, int nullValuesZero, cudaStream_t st)
{
    for (size_t l = 0; l + 1 < start.size(); l++)
    {
        const int n = start[l + 1] - start[l];
        if (n <= 0) continue;
        int blocks = (n + kBcThreads - 1) / kBcThreads;
        if (blocks > 148 * 8) blocks = 148 * 8;
        NB_COUNT_LAUNCH();
        k_bc_level<<<blocks, kBcThreads, 0, st>>>(ops.p + start[l], n, f0, f1, f2, values, nullValuesZero);
    }
}

void RunFlat(const BcFlat &b, double *f0, double *f1, double *f2, const double *values, int nullValuesZero,
             cudaStream_t st)
{
    if (b.nRuns)
    {
        NB_COUNT_LAUNCH();
        k_bc_runs<<<(b.nRuns + kBcThreads / 32 - 1) / (kBcThreads / 32), kBcThreads, 0, st>>>(b.runs.p, b.nRuns, f0, f1, f2,
                                                                                              values);
    }
    else if (b.nOps)
    {
        const int blocks = (b.nOps + kBcThreads - 1) / kBcThreads;
        NB_COUNT_LAUNCH();
        k_bc_level<<<blocks < 148 * 8 ? blocks : 148 * 8, kBcThreads, 0, st>>>(b.ops.p, b.nOps, f0, f1, f2, values,
                                                                              nullValuesZero);
    }
}
} // namespace

void EnforceVelocityDevice(BcReplay &b, double *u, double *v, double *w, const double *prescValues, cudaStream_t st)
{
    if (!u || !v || (b.dim == 3 && !w)) throw InputError("null velocity field");
    // without values the prescribed writes drop out, and with them what the resolved program was resolved from
    if (b.velFlat.ok && (prescValues || b.npresc == 0)) RunFlat(b.velFlat, u, v, w, prescValues, 0, st);
    else RunLevels(b.vel, b.velStart, u, v, w, prescValues, 0, st);
    if (b.ff.nout > 0 && b.ff.aOut > 0.0)
    {
        NB_COUNT_LAUNCH();
        k_bc_outflow<<<1, kFluxThreads, 0, st>>>(b.ff, u, v, w, b.fluxD.p + 2 * (b.ff.nin + b.ff.nout));
    }
    NB_CK(cudaGetLastError());
}

void EnforcePressureDevice(BcReplay &b, double *p, const double *ringValues, cudaStream_t st)
{
    if (!p) throw InputError("null pressure field");
    if (b.presFlat.ok) RunFlat(b.presFlat, p, p, p, ringValues, 1, st);
    else RunLevels(b.pres, b.presStart, p, p, p, ringValues, 1, st);
    NB_CK(cudaGetLastError());
}

} // namespace nb
