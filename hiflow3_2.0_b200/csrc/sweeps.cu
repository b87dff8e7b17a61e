// sweeps.cu -- diagonal kernels and the sync-free level-scheduled sweep.
//
// A level-scheduled triangular solve (lmp/lmatrix_csr_cpu.cc:2295-2392 gives
// the levels; lmp/lpreconditioner_mc_ilup.cc:208-262 the forward / backward
// recurrences) has as many dependent steps as levels -- about 1.5 thousand
// for a 512^2 Q1 grid -- with a few hundred rows each.  One launch per level
// would spend the solve in launch latency, so each sweep is ONE persistent
// launch: warps take chunks of rows in level order from an atomic ticket; a
// chunk never spans two levels, so its rows are independent of one another,
// and every row it depends on belongs to an earlier ticket that a running warp
// already holds.  A row waits (acquire loads, bounded) until the rows it reads
// are published, computes, stores, and publishes itself (release store of the
// sweep's epoch).  Epochs advance by two per apply, so flags never need
// clearing.
#include "b200la.h"
#include "b200la_internal.h"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

using namespace b200;

namespace {

constexpr long long kFlagSpin = 1LL << 22;

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
__global__ void invdiag_kernel(int n, const int *__restrict__ row, const int *__restrict__ col,
                               const T *__restrict__ val, T *__restrict__ out)
{
    // extract_invdiagelements (lmp/lmatrix_csr_cpu.cc:2414-2431)
    for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        T d = T(0);
        for (int j = row[i]; j < row[i + 1]; ++j)
            if (col[j] == i) d = val[j];
        out[i] = T(1) / d;
    }
}

template <typename T>
__global__ void jacobi_kernel(int n, const T *__restrict__ invd, const T *__restrict__ r, T *__restrict__ z,
                              const int *gate)
{
    if (gate_closed(gate)) return;
    for (int i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) z[i] = r[i] * invd[i];
}

struct SyncFreeArgs {
    const int *row, *col;
    const void *val;
    const int2 *chunks;   // {first row, row count}, in dependency order
    int nchunks;
    int lg;               // log2 lanes per row
    const void *r;        // forward: the input
    void *z;              // output (in place)
    const void *d1, *d2;
    unsigned *flags;      // per-row published epoch
    unsigned *sync;       // [epoch base, fwd ticket, bwd ticket, done counter]
    int backward;         // 0 forward, 1 backward
    int sgs;              // 1 MC-SGS recurrences, 0 ILU
    const int *gate;
    int *err;
};

template <typename T>
__global__ void __launch_bounds__(kBlock) syncfree_sweep_kernel(SyncFreeArgs a)
{
    if (gate_closed(a.gate)) return;
    __shared__ unsigned s_epoch;
    if (threadIdx.x == 0) s_epoch = __ldcg(a.sync) + (a.backward ? 2u : 1u);
    __syncthreads();
    const unsigned epoch = s_epoch;
    unsigned *ticket = a.sync + 1 + a.backward;
    const int lane = threadIdx.x & 31;
    const int G = 1 << a.lg;
    const int grp = lane >> a.lg, lg_lane = lane & (G - 1);
    const T *__restrict__ val = static_cast<const T *>(a.val);
    T *z = static_cast<T *>(a.z);
    const T *r = static_cast<const T *>(a.r);
    const T *d1 = static_cast<const T *>(a.d1);
    const T *d2 = static_cast<const T *>(a.d2);
    bool timed_out = false;
    for (;;) {
        int c = 0;
        if (lane == 0) c = (int)atomicAdd(ticket, 1u);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= a.nchunks) break;
        const int2 ch = a.chunks[c];
        const bool active = grp < ch.y;
        const int rr = ch.x + grp;
        T s = T(0);
        if (active) {
            const int j1 = __ldg(a.row + rr + 1);
            for (int j = __ldg(a.row + rr) + lg_lane; j < j1; j += G) {
                const int cc = __ldg(a.col + j);
                long long spin = 0;
                while (ld_acquire(a.flags + cc) != epoch) {
                    // give up (and make every other waiter give up) after a bound
                    if (++spin > kFlagSpin || ((spin & 1023) == 0 && *reinterpret_cast<volatile int *>(a.err))) {
                        timed_out = true;
                        break;
                    }
                }
                s += __ldg(val + j) * __ldcg(z + cc);
            }
        }
        for (int o = G >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (active && lg_lane == 0) {
            T out;
            if (!a.backward) out = a.sgs ? (-r[rr] + s) * d1[rr] : -(-r[rr] + s);
            else out = a.sgs ? (__ldcg(z + rr) * d2[rr] + s) * d1[rr] : (-__ldcg(z + rr) + s) * d1[rr];
            __stcg(z + rr, out);
            st_release(a.flags + rr, epoch);
        }
    }
    if (timed_out) atomicExch(a.err, kDevWaitTimeout);
    // the last block resets the ticket (and advances the epoch after the backward sweep)
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned t = atomicAdd(a.sync + 3, 1u);
        if (t == gridDim.x - 1) {
            a.sync[1 + a.backward] = 0u;
            a.sync[3] = 0u;
            if (a.backward) a.sync[0] = a.sync[0] + 2u;
            __threadfence();
        }
    }
}

// Level sweep in one CTA, for operators with many small levels (the
// level-scheduled ILU(0) of a 2-D grid: ~1,500 levels of ~200 rows).  The
// levels are taken in dependency order, each level's rows by the CTA's 512
// threads, a CTA barrier between levels: no flags, no waits.  The most
// recently solved kLevelRing rows stay in a shared-memory ring, so the
// dependency gathers of a row (on the last few levels) come from shared
// memory; older columns are read from L2.  Forward: rows ascend, a column cc
// of the current level [r0, r1) is in the ring when cc >= r1 - ring (slots of
// rows >= r0 - ring are being rewritten by this level).  Backward: rows
// descend, cc is in the ring when cc < r0 + ring.
constexpr int kLevelRing = 8192;
constexpr int kLevelThreads = 512;
constexpr int kLevelMaxLevels = 24576;   // level offsets kept in shared memory

struct LevelSweepArgs {
    const int *row, *col;
    const void *val;
    const int *off;       // level offsets [nlev + 1] (rows of level l: [off[l], off[l+1]))
    int nlev;
    const void *r;
    void *z;
    const void *d1, *d2;
    int backward, sgs;
    const int *gate;
};

// Row data of one thread in one level, loaded ahead of the level (up to
// kLevelPre entries in registers; longer rows read the rest directly).
constexpr int kLevelPre = 8;
template <typename T>
struct LevelRow {
    int rr, j0, j1;
    int c[kLevelPre];
    T v[kLevelPre];
    T own, e1, e2;   // r_i (forward) or z_i (backward), d1_i, d2_i
};

template <typename T>
__global__ void __launch_bounds__(kLevelThreads) level_sweep_cta_kernel(LevelSweepArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    T *ring = reinterpret_cast<T *>(s_raw);
    int *s_off = reinterpret_cast<int *>(s_raw + kLevelRing * sizeof(T));
    if (gate_closed(a.gate)) return;
    for (int i = threadIdx.x; i <= a.nlev; i += kLevelThreads) {
        s_off[i] = __ldg(a.off + i);
    }
    __syncthreads();
    const T *__restrict__ val = static_cast<const T *>(a.val);
    const T *__restrict__ r = static_cast<const T *>(a.r);
    const T *__restrict__ d1 = static_cast<const T *>(a.d1);
    const T *__restrict__ d2 = static_cast<const T *>(a.d2);
    T *z = static_cast<T *>(a.z);
    const int tid = threadIdx.x, nlev = a.nlev;
    auto level_of = [&](int k) { return a.backward ? nlev - 1 - k : k; };
    // row of this thread in level k (or -1), its row-pointer pair, its entries
    auto first_row = [&](int k) {
        if (k >= nlev) return -1;
        const int l = level_of(k), rr = s_off[l] + tid;
        return rr < s_off[l + 1] ? rr : -1;
    };
    auto load_entries = [&](LevelRow<T> &q) {
#pragma unroll
        for (int e = 0; e < kLevelPre; ++e) {
            if (q.rr >= 0 && q.j0 + e < q.j1) {
                q.c[e] = __ldg(a.col + q.j0 + e);
                q.v[e] = __ldg(val + q.j0 + e);
            }
        }
        if (q.rr >= 0) {
            // the row's own inputs: r_i, or the forward result z_i (written by
            // the previous launch), and the diagonal scalings
            q.own = a.backward ? __ldcg(z + q.rr) : r[q.rr];
            q.e1 = d1 ? d1[q.rr] : T(0);
            q.e2 = (a.sgs && a.backward) ? d2[q.rr] : T(0);
        }
    };
    auto row_value = [&](int rr, int j0, int j1, const int *cp, const T *vp, int r0, int r1, T own, T e1, T e2) {
        T s = T(0);
#pragma unroll
        for (int e = 0; e < kLevelPre; ++e) {
            if (j0 + e < j1) {
                const int cc = cp[e];
                const bool in_ring = a.backward ? cc < r0 + kLevelRing : cc >= r1 - kLevelRing;
                s += vp[e] * (in_ring ? ring[cc & (kLevelRing - 1)] : __ldcg(z + cc));
            }
        }
        for (int j = j0 + kLevelPre; j < j1; ++j) {
            const int cc = __ldg(a.col + j);
            const bool in_ring = a.backward ? cc < r0 + kLevelRing : cc >= r1 - kLevelRing;
            s += __ldg(val + j) * (in_ring ? ring[cc & (kLevelRing - 1)] : __ldcg(z + cc));
        }
        T out;
        if (!a.backward) out = a.sgs ? (-own + s) * e1 : -(-own + s);
        else out = a.sgs ? (own * e2 + s) * e1 : (-own + s) * e1;
        ring[rr & (kLevelRing - 1)] = out;
        __stcg(z + rr, out);
    };
    // software pipeline: entries of level k + 1 and row pointers of level
    // k + 2 are in flight while level k is solved
    LevelRow<T> cur, nxt;
    cur.rr = first_row(0);
    cur.j0 = cur.rr >= 0 ? __ldg(a.row + cur.rr) : 0;
    cur.j1 = cur.rr >= 0 ? __ldg(a.row + cur.rr + 1) : 0;
    load_entries(cur);
    nxt.rr = first_row(1);
    nxt.j0 = nxt.rr >= 0 ? __ldg(a.row + nxt.rr) : 0;
    nxt.j1 = nxt.rr >= 0 ? __ldg(a.row + nxt.rr + 1) : 0;
    for (int k = 0; k < nlev; ++k) {
        const int l = level_of(k), r0 = s_off[l], r1 = s_off[l + 1];
        const int r2 = first_row(k + 2);
        const int p0 = r2 >= 0 ? __ldg(a.row + r2) : 0, p1 = r2 >= 0 ? __ldg(a.row + r2 + 1) : 0;
        load_entries(nxt);
        if (cur.rr >= 0) row_value(cur.rr, cur.j0, cur.j1, cur.c, cur.v, r0, r1, cur.own, cur.e1, cur.e2);
        // rows of a level beyond the first kLevelThreads (no look-ahead)
        for (int rr = r0 + tid + kLevelThreads; rr < r1; rr += kLevelThreads) {
            LevelRow<T> q;
            q.rr = rr;
            q.j0 = __ldg(a.row + rr);
            q.j1 = __ldg(a.row + rr + 1);
            load_entries(q);
            row_value(rr, q.j0, q.j1, q.c, q.v, r0, r1, q.own, q.e1, q.e2);
        }
        __syncthreads();
        cur = nxt;
        nxt.rr = r2;
        nxt.j0 = p0;
        nxt.j1 = p1;
    }
}

// The level sweep with a deeper look-ahead through the async-copy engine, for
// operators that the packed stream below does not take.
// At set-up every row of L / U is packed into kp fixed slots (columns and
// values, the entry count beside).  Each thread copies its row of level
// k + kStages - 1 (packed entries, count, own input and scalings) into a
// shared-memory stage with cp.async while level k is solved, so the loads of
// a level arrive kStages - 1 levels early and only the ring gathers, the
// solve and the level barrier remain on the critical path.
constexpr int kStages = 4;
constexpr int kRingStaged = 4096;
constexpr int kStagedMaxLevels = 4096;
constexpr int kStagedSlots = 4;    // packed entries per row (rows of L and U with at most this many)

struct LevelStagedArgs {
    const int *pcol;      // packed columns [n][kp]
    const void *pval;     // packed values [n][kp]
    const int *pcnt;      // entries per row
    const int *off;
    int nlev, n;
    const void *r;
    void *z;
    const void *d1, *d2;
    int backward, sgs;
    const int *gate;
};

__device__ __forceinline__ void cp_async(void *dst, const void *src, int bytes)
{
    const unsigned d = smem_u32(dst);
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
    else if (bytes == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, int KP>
struct StageRec {
    int col[KP];
    T val[KP];
    T own, e1, e2;
    int cnt;
};

template <typename T, int KP>
__global__ void __launch_bounds__(kLevelThreads) level_sweep_staged_kernel(LevelStagedArgs a)
{
    // one thread per row of the largest level (blockDim.x <= kLevelThreads):
    // idle warps would only lengthen every level's barrier
    const int NT = blockDim.x;
    extern __shared__ __align__(16) unsigned char s_raw[];
    using Rec = StageRec<T, KP>;
    Rec *stage = reinterpret_cast<Rec *>(s_raw);                             // [kStages][NT]
    T *ring = reinterpret_cast<T *>(s_raw + sizeof(Rec) * kStages * NT);
    int *s_off = reinterpret_cast<int *>(ring + kRingStaged);
    if (gate_closed(a.gate)) return;
    for (int i = threadIdx.x; i <= a.nlev; i += NT) s_off[i] = __ldg(a.off + i);
    __syncthreads();
    const int tid = threadIdx.x, nlev = a.nlev;
    const T *pval = static_cast<const T *>(a.pval);
    const T *r = static_cast<const T *>(a.r);
    const T *d1 = static_cast<const T *>(a.d1);
    const T *d2 = static_cast<const T *>(a.d2);
    T *z = static_cast<T *>(a.z);
    const bool need_e1 = a.backward || a.sgs, need_e2 = a.backward && a.sgs;
    auto level_of = [&](int k) { return a.backward ? nlev - 1 - k : k; };
    // this thread's row of level k into stage k % kStages (one commit group per level)
    auto issue = [&](int k) {
        if (k < nlev) {
            const int l = level_of(k), rr = s_off[l] + tid;
            if (rr < s_off[l + 1]) {
                Rec &q = stage[(k % kStages) * NT + tid];
#pragma unroll
                for (int b = 0; b < KP * 4; b += 16) cp_async(reinterpret_cast<char *>(q.col) + b,
                                                              reinterpret_cast<const char *>(a.pcol + (size_t)rr * KP) + b, 16);
#pragma unroll
                for (int b = 0; b < KP * (int)sizeof(T); b += 16)
                    cp_async(reinterpret_cast<char *>(q.val) + b, reinterpret_cast<const char *>(pval + (size_t)rr * KP) + b,
                             16);
                cp_async(&q.cnt, a.pcnt + rr, 4);
                cp_async(&q.own, (a.backward ? static_cast<const T *>(z) : r) + rr, (int)sizeof(T));
                if (need_e1) cp_async(&q.e1, d1 + rr, (int)sizeof(T));
                if (need_e2) cp_async(&q.e2, d2 + rr, (int)sizeof(T));
            }
        }
        cp_async_commit();
    };
    auto solve = [&](int rr, const int *cols, const T *vals, int cnt, T own, T e1, T e2, int r0, int r1) {
        T s = T(0);
#pragma unroll
        for (int e = 0; e < KP; ++e) {
            if (e < cnt) {
                const int cc = cols[e];
                const bool in_ring = a.backward ? cc < r0 + kRingStaged : cc >= r1 - kRingStaged;
                s += vals[e] * (in_ring ? ring[cc & (kRingStaged - 1)] : __ldcg(z + cc));
            }
        }
        T out;
        if (!a.backward) out = a.sgs ? (-own + s) * e1 : -(-own + s);
        else out = a.sgs ? (own * e2 + s) * e1 : (-own + s) * e1;
        ring[rr & (kRingStaged - 1)] = out;
        __stcg(z + rr, out);
    };
#pragma unroll
    for (int k = 0; k < kStages - 1; ++k) issue(k);
    for (int k = 0; k < nlev; ++k) {
        issue(k + kStages - 1);
        cp_async_wait<kStages - 1>();
        const int l = level_of(k), r0 = s_off[l], r1 = s_off[l + 1];
        const int rr = r0 + tid;
        if (rr < r1) {
            const Rec &q = stage[(k % kStages) * NT + tid];
            solve(rr, q.col, q.val, q.cnt, q.own, need_e1 ? q.e1 : T(0), need_e2 ? q.e2 : T(0), r0, r1);
        }
        // rows of a level beyond the first NT: read directly
        for (int r2 = rr + NT; r2 < r1; r2 += NT) {
            int cols[KP];
            T vals[KP];
#pragma unroll
            for (int e = 0; e < KP; ++e) {
                cols[e] = __ldg(a.pcol + (size_t)r2 * KP + e);
                vals[e] = __ldg(pval + (size_t)r2 * KP + e);
            }
            const T own = a.backward ? __ldcg(z + r2) : r[r2];
            solve(r2, cols, vals, __ldg(a.pcnt + r2), own, need_e1 ? d1[r2] : T(0), need_e2 ? d2[r2] : T(0), r0, r1);
        }
        __syncthreads();
    }
    cp_async_wait<0>();
}

// Pack the rows of a CSR into kp fixed slots (columns, values; unused slots
// column 0, value 0) with the entry count beside.
template <typename T>
__global__ void pack_rows_kernel(int n, int kp, const int *__restrict__ row, const int *__restrict__ col,
                                 const T *__restrict__ val, int *__restrict__ pcol, T *__restrict__ pval,
                                 int *__restrict__ pcnt)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int b = row[i], e = row[i + 1];
        for (int k = 0; k < kp; ++k) {
            const bool in = b + k < e;
            pcol[(size_t)i * kp + k] = in ? col[b + k] : 0;
            pval[(size_t)i * kp + k] = in ? val[b + k] : T(0);
        }
        pcnt[i] = e - b;
    }
}

constexpr size_t kStagedSmemCap = 226 * 1024;   // opt-in shared memory per CTA on sm_100 (227 KB), less the static part

template <typename T, int KP>
size_t staged_smem(int nlev, int NT = kLevelThreads)
{
    return sizeof(StageRec<T, KP>) * kStages * NT + sizeof(T) * kRingStaged + sizeof(int) * (nlev + 1);
}


// The level sweep on a packed stream of the factor, both directions in one
// launch.  At set-up the rows of L and U are packed, in dependency order, into
// tiles of at most pack_rows(KP) consecutive rows of one level: a 16-byte
// header (first row, rows) and one record per row -- the values, where their
// vector entries lie (16-bit byte offsets) and the diagonal scalings.
// Producer warps bring each tile and the rows' own inputs (r, then the forward
// result) into a ring of shared-memory stages by bulk copies, several tiles
// ahead; the other warps solve one row per thread.  The results of the last
// kPackRing rows stay in shared memory, where the next levels gather them;
// entries further back (the identity rows of level 0, for instance) are copied
// ahead by the producer into slots of the stage.
//   The sweep is a serial chain of levels: what bounds it is the instruction
// stream of one level, not its bytes (about 60 per FP64 row of four entries).
// So a level's records are read while the level before it is solved, its
// header a level earlier still, a watching warp does the waiting for tiles, and
// between two barriers stand one gather per entry, the products in column order
// and the store into the ring.  Four producer warps: one needs about 1,000
// cycles per tile.  One CTA: across SMs every level would wait for a cluster
// barrier and for remote shared memory.
//   Measured (one apply, both directions; before: one cp.async look-ahead per
// thread for rows of up to four entries, a register look-ahead for longer
// ones): 2-D 512^2 ILU(0), 1,537 levels, FP64 2,470 -> 710 us (0.23 us per
// level); 256^2 1,060 -> 300 us, FP32 245 us; 150^2 ILU(1) 1,880 -> 410 us.
constexpr int kPackMaxRows = 512;
constexpr int pack_rows(int kp) { return kp == 4 ? kPackMaxRows : kp == 8 ? 256 : 192; }   // rows of a tile
constexpr int kPackMaxStages = 8;
constexpr int kPackMinStages = 4;
constexpr int kPackRing = 4096;    // at least kPackMaxStages tiles, so that what lies further back is solved
constexpr int kPackProducers = 4;   // producer warps
static_assert(kPackProducers <= kPackMinStages, "two warps must not wait for the same stage's phases at once");
constexpr int kPackFar = 32;       // far entries of a tile
constexpr int kPackMaxEntries = 16;
constexpr size_t kPackSmemCap = 225 * 1024;   // of the 227 KB a CTA can have, less the static part
static_assert(kPackRing >= kPackMaxStages * kPackMaxRows, "far entries must be solved when their tile is issued");

struct alignas(16) PackTile {
    int row0, m;
    unsigned off16;          // the tile's packed bytes start at 16 * off16
    int far0, nfar;          // its far columns
    int pad[3];
};

struct PackedSweepArgs {
    const PackTile *tiles;          // forward tiles, then backward tiles
    const unsigned char *pack;
    const int *far;                 // far columns of all tiles, and their number
    int nf, nt;                     // forward tiles, all tiles
    int nfar, n, stages, stage_bytes, own_off;
    const void *r;
    void *z;
    const int *gate;
    int *err;
};

// Row record: KP values, KP offsets, one scaling (two for SGS); padded so that
// the eight lanes of a 16-byte shared-memory phase fall on different banks.
template <typename T, int KP, bool SGS>
struct PackRec {
    static constexpr int scal = KP * (int)sizeof(T) + 2 * KP;
    static constexpr int used = (scal + (SGS ? 2 : 1) * (int)sizeof(T) + 15) & ~15;
    static constexpr int bytes = (used / 16) % 2 == 1 ? used : used + 16;
};
// shared memory before the stages: the ring, a zero entry, the stages' far entries
template <typename T>
__host__ __device__ constexpr int pack_far_off() { return kPackRing * (int)sizeof(T) + 16; }
template <typename T>
__host__ __device__ constexpr int pack_head_bytes()
{
    return pack_far_off<T>() + kPackMaxStages * kPackFar * (int)sizeof(T);
}
static_assert(pack_head_bytes<double>() <= 65536, "16-bit offsets");

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// arrives when the calling thread's cp.async copies so far have landed
__device__ __forceinline__ void mbar_arrive_cp_async(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <typename T>
__device__ __forceinline__ void cp_async_one(void *dst, const T *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(sizeof(T)) : "memory");
}

struct PackedShared {
    uint64_t full[kPackMaxStages], empty[kPackMaxStages], fwd_done;
    int fail;
};

// The barrier between two tiles, of the solving warps and the watching warp.
__device__ __forceinline__ void packed_barrier(int threads)
{
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

template <typename T, int KP>
struct PackedRow {
    T v[KP];
    unsigned ix[KP / 2];   // byte offsets of the row's vector entries, in pairs
    int at[KP];            // and unpacked
    T own, e1, e2;
};

// One direction of the sweep, by the solving threads: cnt tiles, the first of
// them in stage `stg`.  A tile may be read from the barrier before the tile
// ahead of it on (the watching warp has seen it arrive).
template <typename T, int KP, bool SGS, bool BWD>
__device__ __forceinline__ void packed_phase(const PackedSweepArgs &a, unsigned char *smem, const PackedShared &sh, int cnt,
                                             int &stg, int NT)
{
    using Rec = PackRec<T, KP, SGS>;
    constexpr int R = Rec::bytes;
    const int tid = threadIdx.x, S = a.stages;
    T *z = static_cast<T *>(a.z);
    const T *vec = BWD ? z : static_cast<const T *>(a.r);
    constexpr unsigned W = 16 / sizeof(T) - 1;
    const unsigned vsh = (unsigned)(reinterpret_cast<uintptr_t>(vec) / sizeof(T)) & W;   // first element in its 16 bytes
    const unsigned char *stages = smem + pack_head_bytes<T>();
    const unsigned char *rec_at = stages + 16 + tid * R;
    const T *own_at = reinterpret_cast<const T *>(stages + a.own_off) + tid;
    auto next = [&](int s) { return s + 1 == S ? 0 : s + 1; };
    auto header = [&](int s) { return *reinterpret_cast<const int2 *>(stages + s * a.stage_bytes); };
    // after a wait has run out no tile is read: its bytes may not have arrived
    // (the flag is read with a header and looked at a level later)
    auto failed = [&]() { return *static_cast<const volatile int *>(&sh.fail); };
    auto record = [&](PackedRow<T, KP> &q, int s, int2 h) {
        if (tid >= h.y) return;
        const uint4 *p = reinterpret_cast<const uint4 *>(rec_at + s * a.stage_bytes);
        uint4 w[Rec::used / 16];
#pragma unroll
        for (int i = 0; i < Rec::used / 16; ++i) w[i] = p[i];
        const unsigned *u = reinterpret_cast<const unsigned *>(w);
        auto get = [&](int byte) -> T {
            if constexpr (sizeof(T) == 8) return __hiloint2double((int)u[byte / 4 + 1], (int)u[byte / 4]);
            else return __uint_as_float(u[byte / 4]);
        };
#pragma unroll
        for (int e = 0; e < KP; ++e) q.v[e] = get(e * (int)sizeof(T));
#pragma unroll
        for (int e = 0; e < KP / 2; ++e) q.ix[e] = u[KP * (int)sizeof(T) / 4 + e];
        if (BWD || SGS) q.e1 = get(Rec::scal);
        if (BWD && SGS) q.e2 = get(Rec::scal + (int)sizeof(T));
        q.own = reinterpret_cast<const T *>(reinterpret_cast<const unsigned char *>(own_at) +
                                            s * a.stage_bytes)[(vsh + (unsigned)h.x) & W];
    };
    // (apart from the loads: it waits for them)
    auto unpack = [&](PackedRow<T, KP> &q) {
#pragma unroll
        for (int e = 0; e < KP; ++e) q.at[e] = (int)(e & 1 ? q.ix[e / 2] >> 16 : q.ix[e / 2] & 0xffffu);
    };
    int s1 = next(stg), s2 = next(s1);
    packed_barrier(NT + 32);   // the first two tiles are there
    int fn = failed();
    int2 hc = header(stg), hn = cnt > 1 ? header(s1) : make_int2(0, 0);
    if (fn) hc.y = 0;
    PackedRow<T, KP> ra, rb;
    record(ra, stg, hc);
    unpack(ra);
    auto step = [&](PackedRow<T, KP> &cur, PackedRow<T, KP> &nxt, int k) {
        const bool active = tid < hc.y;
        T g[KP];
#pragma unroll
        for (int e = 0; e < KP; ++e) g[e] = active ? *reinterpret_cast<const T *>(smem + cur.at[e]) : T(0);
        if (fn) hn.y = 0;
        record(nxt, s1, hn);
        T s = T(0);
#pragma unroll
        for (int e = 0; e < KP; ++e) s += cur.v[e] * g[e];
        T out;
        if (!BWD) out = SGS ? (-cur.own + s) * cur.e1 : -(-cur.own + s);
        else out = SGS ? (cur.own * cur.e2 + s) * cur.e1 : (-cur.own + s) * cur.e1;
        if (active) {
            const int rr = hc.x + tid;
            reinterpret_cast<T *>(smem)[rr & (kPackRing - 1)] = out;
            z[rr] = out;
        }
        unpack(nxt);
        if (!BWD && k + 1 == cnt) asm volatile("fence.proxy.async.global;" ::: "memory");   // z before its bulk copies
        packed_barrier(NT + 32);
        hc = hn;
        hn = k + 2 < cnt ? header(s2) : make_int2(0, 0);
        fn = failed();
        s1 = s2;
        s2 = next(s2);
    };
    for (int k = 0; k < cnt; k += 2) {
        step(ra, rb, k);
        if (k + 1 < cnt) step(rb, ra, k + 1);
    }
    stg = (stg + cnt) % S;
}

template <typename T, int KP, bool SGS>
__global__ void __launch_bounds__(pack_rows(KP) + 32 * (1 + kPackProducers), 1)
    level_sweep_packed_kernel(PackedSweepArgs a)
{
    if (gate_closed(a.gate)) return;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ PackedShared sh;
    const int tid = threadIdx.x, NT = blockDim.x - 32 * (1 + kPackProducers), S = a.stages, nf = a.nf, nt = a.nt;
    if (tid == 0) {
        for (int i = 0; i < kPackMaxStages; ++i) {
            mbar_init(&sh.full[i], a.nfar ? 1 + 32 : 1);
            mbar_init(&sh.empty[i], 1);
        }
        mbar_init(&sh.fwd_done, 1);
        fence_mbar_init();
        sh.fail = 0;
        *reinterpret_cast<T *>(s_raw + kPackRing * sizeof(T)) = T(0);
    }
    __syncthreads();
    if (tid < NT) {
        int stg = 0;
        packed_phase<T, KP, SGS, false>(a, s_raw, sh, nf, stg, NT);
        packed_phase<T, KP, SGS, true>(a, s_raw, sh, nt - nf, stg, NT);
        return;
    }
    // bounded waits: after one has run out (reported in *err) nothing waits any more
    auto wait = [&](uint64_t *bar, unsigned parity) {
        if (mbar_try_wait(bar, parity)) return true;
        volatile int *fail = &sh.fail;
        if (!*fail && !mbar_wait_bounded(bar, parity, a.err)) *fail = 1;
        return *fail == 0;
    };
    const int lane = tid & 31, w = ((tid - NT) >> 5) - 1;
    if (w < 0) {
        // Watching warp: it meets the barrier after a tile once the tile two
        // ahead has arrived, and hands the solved tile's stage back, so that
        // the solving warps look at no arrival barrier themselves.
        for (int k0 = 0, k1 = nf; k0 < nt; k0 = k1, k1 = nt) {
            for (int q = k0; q < min(k0 + 2, k1); ++q) wait(&sh.full[q % S], (unsigned)(q / S) & 1u);
            packed_barrier(NT + 32);
            int s = k0 % S, s2 = (k0 + 2) % S;
            unsigned p2 = (unsigned)((k0 + 2) / S) & 1u;
            for (int k = k0; k < k1; ++k) {
                if (k + 2 < k1) wait(&sh.full[s2], p2);
                packed_barrier(NT + 32);
                if (lane == 0) mbar_arrive(&sh.empty[s]);
                if (++s == S) s = 0;
                if (++s2 == S) {
                    s2 = 0;
                    p2 ^= 1u;
                }
            }
            if (k1 == nf && lane == 0) mbar_arrive(&sh.fwd_done);
        }
        return;
    }
    // Producer warps, tile k by warp k % kPackProducers; descriptors and far
    // columns are read ahead (a load per tile on its own path would put a
    // memory round trip into every level).
    const uint64_t pol = l2_policy(0);
    constexpr int W = 16 / (int)sizeof(T) - 1;
    T *z = static_cast<T *>(a.z);
    auto tile_at = [&](int k) { return a.tiles[min(k, nt - 1)]; };
    auto far_at = [&](const PackTile &t) { return lane < t.nfar ? __ldg(a.far + t.far0 + lane) : 0; };
    PackTile t = tile_at(w), t1 = tile_at(w + kPackProducers);
    int f = far_at(t), k = w;
    bool backward = false;
    for (; k < nt; k += kPackProducers) {
        const PackTile t2 = tile_at(k + 2 * kPackProducers);
        const int f1 = far_at(t1), s = k % S;
        bool ok = k < S || wait(&sh.empty[s], (unsigned)(k / S - 1) & 1u);
        if (!backward && k >= nf) {   // the backward inputs are the forward results
            ok = wait(&sh.fwd_done, 0u) && ok;
            backward = true;
        }
        if (!__all_sync(0xffffffffu, ok)) break;
        unsigned char *st = s_raw + pack_head_bytes<T>() + (size_t)s * a.stage_bytes;
        if (lane < t.nfar) cp_async_one(reinterpret_cast<T *>(s_raw + pack_far_off<T>()) + s * kPackFar + lane, z + f);
        if (lane == 0) {
            // own inputs: the 16-byte units around [row0, row0 + m); at the
            // vector's ragged ends the elements inside it one by one
            const T *vec = backward ? z : static_cast<const T *>(a.r);
            const int sft = (int)(((unsigned)(reinterpret_cast<uintptr_t>(vec) / sizeof(T)) + (unsigned)t.row0) & W);
            int q0 = t.row0 - sft, q1 = q0 + ((sft + t.m + W) & ~W);
            T *own = reinterpret_cast<T *>(st + a.own_off) + sft - t.row0;   // own[i] for row i
            if (q0 < 0 || q1 > a.n) {
                if (q0 < 0) q0 += W + 1;
                if (q1 > a.n) q1 -= W + 1;
                if (q1 < q0) q0 = q1 = t.row0 + t.m;
                for (int i = t.row0; i < t.row0 + t.m; ++i)
                    if (i < q0 || i >= q1) own[i] = __ldcg(vec + i);
            }
            const unsigned ob = (unsigned)(q1 - q0) * (unsigned)sizeof(T);
            const unsigned bytes = 16u + (unsigned)(t.m * PackRec<T, KP, SGS>::bytes);
            mbar_arrive_expect_tx(&sh.full[s], bytes + ob);
            bulk_g2s(st, a.pack + 16 * (size_t)t.off16, bytes, &sh.full[s], pol);
            if (ob) bulk_g2s(own + q0, vec + q0, ob, &sh.full[s], pol);
        }
        __syncwarp();   // no lane waits for a later stage while lane 0 has yet to issue this tile
        if (a.nfar) mbar_arrive_cp_async(&sh.full[s]);
        t = t1;
        t1 = t2;
        f = f1;
    }
    if (k < nt)   // a wait has run out: leave none of this warp's copies in flight
        for (int q = w; q < k; q += kPackProducers)
            if (q >= k - S) mbar_wait_bounded(&sh.full[q % S], (unsigned)(q / S) & 1u, a.err);
}

// Set-up: the far columns of every tile (fill = 0: counted into nfar[], fill =
// 1: listed at far0 in row order), and the packed tiles.  One warp per tile.
__device__ __forceinline__ bool pack_is_far(bool bwd, int r0, int r1, int c)
{
    return (bwd ? c - r0 + 1 : r1 - c) > kPackRing;
}
__global__ void pack_far_kernel(int nt, int nf, PackTile *tiles, const int *__restrict__ rl, const int *__restrict__ cl,
                                const int *__restrict__ ru, const int *__restrict__ cu, int fill, int *far)
{
    const int k = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (k >= nt) return;
    const bool bwd = k >= nf;
    const int *row = bwd ? ru : rl, *col = bwd ? cu : cl;
    const int r0 = tiles[k].row0, r1 = r0 + tiles[k].m, far0 = tiles[k].far0, end = row[r1];
    int c = 0;
    for (int j0 = row[r0]; j0 < end; j0 += 32) {
        const int cj = j0 + lane < end ? col[j0 + lane] : 0;
        const bool is = j0 + lane < end && pack_is_far(bwd, r0, r1, cj);
        const unsigned b = __ballot_sync(0xffffffffu, is);
        if (fill && is) far[far0 + c + __popc(b & ((1u << lane) - 1u))] = cj;
        c += __popc(b);
    }
    if (!fill && lane == 0) tiles[k].nfar = c;
}

template <typename T, int KP, bool SGS>
__global__ void pack_tiles_kernel(int nt, int nf, const PackTile *__restrict__ tiles, const int *__restrict__ rl,
                                  const int *__restrict__ cl, const T *__restrict__ vl, const int *__restrict__ ru,
                                  const int *__restrict__ cu, const T *__restrict__ vu, const T *__restrict__ d1,
                                  const T *__restrict__ d2, int stages, unsigned char *__restrict__ pack)
{
    const int k = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (k >= nt) return;
    const bool bwd = k >= nf;
    const PackTile t = tiles[k];
    const int *row = bwd ? ru : rl, *col = bwd ? cu : cl;
    const T *val = bwd ? vu : vl;
    unsigned char *st = pack + 16 * (size_t)t.off16;
    if (lane == 0) *reinterpret_cast<int4 *>(st) = make_int4(t.row0, t.m, 0, 0);
    const int slot0 = pack_far_off<T>() + (k % stages) * kPackFar * (int)sizeof(T);
    int far_before = 0;   // far entries of the rows of earlier passes
    for (int i0 = 0; i0 < t.m; i0 += 32) {
        const int i = i0 + lane, rr = t.row0 + i;
        const int b = i < t.m ? row[rr] : 0, cnt = i < t.m ? row[rr + 1] - b : 0;
        int fc = 0;
        for (int e = 0; e < cnt; ++e) fc += pack_is_far(bwd, t.row0, t.row0 + t.m, col[b + e]);
        int incl = fc;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        int slot = far_before + incl - fc;
        far_before += __shfl_sync(0xffffffffu, incl, 31);
        if (i < t.m) {
            unsigned char *q = st + 16 + (size_t)i * PackRec<T, KP, SGS>::bytes;
            T *v = reinterpret_cast<T *>(q);
            unsigned short *ix = reinterpret_cast<unsigned short *>(q + KP * sizeof(T));
            for (int e = 0; e < KP; ++e) {
                v[e] = e < cnt ? val[b + e] : T(0);
                int off = kPackRing * (int)sizeof(T);   // the zero entry
                if (e < cnt) {
                    const int c = col[b + e];
                    off = pack_is_far(bwd, t.row0, t.row0 + t.m, c) ? slot0 + (slot++) * (int)sizeof(T)
                                                                    : (c & (kPackRing - 1)) * (int)sizeof(T);
                }
                ix[e] = (unsigned short)off;
            }
            T *sc = reinterpret_cast<T *>(q + PackRec<T, KP, SGS>::scal);
            sc[0] = d1[rr];
            if (SGS) sc[1] = d2[rr];
        }
    }
}

template <typename T, int KP>
cudaError_t packed_attr()
{
    cudaError_t e = cudaFuncSetAttribute(level_sweep_packed_kernel<T, KP, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPackSmemCap);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(level_sweep_packed_kernel<T, KP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kPackSmemCap);
}

}  // namespace

namespace b200 {

cudaError_t sweeps_configure()
{
    cudaError_t e;
    // the largest stage set a plan may use (its CTA size and level count are
    // checked against kStagedSmemCap at set-up)
    if ((e = cudaFuncSetAttribute(level_sweep_staged_kernel<double, kStagedSlots>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::min(staged_smem<double, kStagedSlots>(kStagedMaxLevels), kStagedSmemCap))) ||
        (e = cudaFuncSetAttribute(level_sweep_staged_kernel<float, kStagedSlots>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::min(staged_smem<float, kStagedSlots>(kStagedMaxLevels), kStagedSmemCap))))
        return e;
    if ((e = packed_attr<double, 4>()) || (e = packed_attr<double, 8>()) || (e = packed_attr<double, 16>()) ||
        (e = packed_attr<float, 4>()) || (e = packed_attr<float, 8>()) || (e = packed_attr<float, 16>()))
        return e;
    e = cudaFuncSetAttribute(level_sweep_cta_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kLevelRing * sizeof(double) + sizeof(int) * (kLevelMaxLevels + 1)));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(level_sweep_cta_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kLevelRing * sizeof(float) + sizeof(int) * (kLevelMaxLevels + 1)));
}

cudaError_t launch_invdiag(int dtype, int n, const int *row, const int *col, const void *val, void *out,
                           cudaStream_t st)
{
    const int g = std::max(1, std::min((n + kBlock - 1) / kBlock, 148 * 8));
    if (dtype == B200LA_F64)
        invdiag_kernel<double><<<g, kBlock, 0, st>>>(n, row, col, (const double *)val, (double *)out);
    else
        invdiag_kernel<float><<<g, kBlock, 0, st>>>(n, row, col, (const float *)val, (float *)out);
    return cudaGetLastError();
}

cudaError_t launch_jacobi(int dtype, int n, const void *invd, const void *r, void *z, const int *gate,
                          cudaStream_t st)
{
    const int g = std::max(1, std::min((n + kBlock * 4 - 1) / (kBlock * 4), 148 * 8));
    if (dtype == B200LA_F64)
        jacobi_kernel<double><<<g, kBlock, 0, st>>>(n, (const double *)invd, (const double *)r, (double *)z, gate);
    else
        jacobi_kernel<float><<<g, kBlock, 0, st>>>(n, (const float *)invd, (const float *)r, (float *)z, gate);
    return cudaGetLastError();
}

}  // namespace b200

// Host side: chunk lists and launches.

struct SyncFreePlan {
    int2 *fwd = nullptr, *bwd = nullptr;
    int nf = 0, nb = 0;
    int lg_l = 0, lg_u = 0;
    int *lev_off = nullptr;   // single-CTA level sweep: level offsets (null: chunk tickets)
    int nlev = 0;
    // look-ahead variant (staged_threads > 0, the CTA's): rows of L / U in kStagedSlots slots
    int staged_threads = 0;
    int *pcol[2] = {nullptr, nullptr}, *pcnt[2] = {nullptr, nullptr};
    void *pval[2] = {nullptr, nullptr};
    // packed variant (kp > 0): the tiles and the packed stream of both sweeps
    int kp = 0, threads = 0, nf_tiles = 0, nt_tiles = 0, stages = 0, stage_bytes = 0, own_off = 0, nfar = 0;
    PackTile *ptiles = nullptr;
    int *far = nullptr;
    unsigned char *pack = nullptr;
};

static int lanes_for(const b200la_csr *M)
{
    const double mean = M->n ? (double)M->nnz / M->n : 0.0;
    int lg = 0;
    while (lg < 5 && (double)(1 << lg) < mean) ++lg;
    return lg;
}

// The packed plan of P's sweeps; plan->kp stays 0 when the operator does not
// fit it (rows too long, too many far columns in a tile).
template <typename T, int KP, bool SGS>
static cudaError_t packed_setup(b200la_ctx *ctx, const b200la_precond *P, SyncFreePlan *plan)
{
    constexpr int R = PackRec<T, KP, SGS>::bytes, cap = pack_rows(KP);
    std::vector<PackTile> tiles;
    size_t off = 0;
    int widest = 1;
    auto add = [&](int r0, int m) {
        PackTile t{};
        t.row0 = r0;
        t.m = m;
        t.off16 = (unsigned)(off / 16);
        off += 16 + (size_t)m * R;
        widest = std::max(widest, m);
        tiles.push_back(t);
    };
    for (int l = 0; l < P->nblocks; ++l)
        for (int r = P->block_off[l]; r < P->block_off[l + 1]; r += cap) add(r, std::min(cap, P->block_off[l + 1] - r));
    const int nf = (int)tiles.size();
    for (int l = P->nblocks - 1; l >= 0; --l)   // rows strictly descending by tile
        for (int e = P->block_off[l + 1]; e > P->block_off[l]; e -= cap) {
            const int r = std::max(P->block_off[l], e - cap);
            add(r, e - r);
        }
    if (off / 16 > 0xffffffffull) return cudaSuccess;
    const int nt = (int)tiles.size(), threads = (widest + 31) / 32 * 32;
    const int own_off = 16 + threads * R, stage = (own_off + (int)sizeof(T) * threads + 32 + 127) & ~127;
    const int stages = (int)std::min<size_t>(kPackMaxStages, (kPackSmemCap - pack_head_bytes<T>()) / stage);
    if (stages < kPackMinStages) return cudaSuccess;
    cudaError_t e;
    const size_t tb = sizeof(PackTile) * nt;
    if ((e = cudaMalloc(&plan->ptiles, tb)) || (e = setup_copy(ctx->stream, plan->ptiles, tiles.data(), tb)))
        return e;
    pack_far_kernel<<<(nt + 3) / 4, 128, 0, ctx->stream>>>(nt, nf, plan->ptiles, P->L->row, P->L->col, P->U->row,
                                                           P->U->col, 0, nullptr);
    if ((e = cudaGetLastError()) ||
        (e = cudaMemcpyAsync(tiles.data(), plan->ptiles, tb, cudaMemcpyDeviceToHost, ctx->stream)) ||
        (e = cudaStreamSynchronize(ctx->stream)))
        return e;
    long long nfar = 0;
    for (PackTile &t : tiles) {
        if (t.nfar > kPackFar || nfar > INT_MAX - 64) return cudaSuccess;
        t.far0 = (int)nfar;
        nfar += t.nfar;
    }
    if ((e = setup_copy(ctx->stream, plan->ptiles, tiles.data(), tb)) ||
        (e = cudaMalloc(&plan->far, sizeof(int) * std::max<long long>(nfar, 1))) ||
        (e = cudaMalloc(&plan->pack, std::max<size_t>(off, 16))))
        return e;
    pack_far_kernel<<<(nt + 3) / 4, 128, 0, ctx->stream>>>(nt, nf, plan->ptiles, P->L->row, P->L->col, P->U->row,
                                                           P->U->col, 1, plan->far);
    pack_tiles_kernel<T, KP, SGS><<<(nt + 3) / 4, 128, 0, ctx->stream>>>(
        nt, nf, plan->ptiles, P->L->row, P->L->col, (const T *)P->L->val, P->U->row, P->U->col, (const T *)P->U->val,
        (const T *)P->iDv, (const T *)P->Dv, stages, plan->pack);
    if ((e = cudaGetLastError()) || (e = cudaStreamSynchronize(ctx->stream))) return e;
    plan->threads = threads;
    plan->nf_tiles = nf;
    plan->nt_tiles = nt;
    plan->stages = stages;
    plan->stage_bytes = stage;
    plan->own_off = own_off;
    plan->nfar = (int)nfar;
    plan->kp = KP;
    return cudaSuccess;
}

template <typename T, int KP, bool SGS>
static cudaError_t packed_launch(const SyncFreePlan *plan, const PackedSweepArgs &a, cudaStream_t st)
{
    const size_t sm = pack_head_bytes<T>() + (size_t)plan->stages * plan->stage_bytes;
    level_sweep_packed_kernel<T, KP, SGS><<<1, plan->threads + 32 * (1 + kPackProducers), sm, st>>>(a);
    return cudaGetLastError();
}

// f(type, entries, sgs) for the packed kernel instance of P with kp entries per row
template <class F>
static cudaError_t packed_dispatch(const b200la_precond *P, int kp, F f)
{
    auto by_kp = [&](auto t, auto sgs) {
        using I4 = std::integral_constant<int, 4>;
        using I8 = std::integral_constant<int, 8>;
        using I16 = std::integral_constant<int, 16>;
        return kp == 4 ? f(t, I4(), sgs) : kp == 8 ? f(t, I8(), sgs) : f(t, I16(), sgs);
    };
    auto by_type = [&](auto sgs) { return P->dtype == B200LA_F64 ? by_kp(double(), sgs) : by_kp(float(), sgs); };
    return P->kind == B200LA_PRECOND_MCSGS ? by_type(std::true_type()) : by_type(std::false_type());
}

// Rows of L and U in slots, for the look-ahead variant.
template <typename T>
static cudaError_t staged_setup(b200la_ctx *ctx, const b200la_precond *P, SyncFreePlan *plan, int threads)
{
    const size_t n = (size_t)P->n;
    cudaError_t e = cudaSuccess;
    for (int m = 0; m < 2 && e == cudaSuccess; ++m) {
        const b200la_csr *M = m ? P->U : P->L;
        if ((e = cudaMalloc(&plan->pcol[m], sizeof(int) * kStagedSlots * n)) ||
            (e = cudaMalloc(&plan->pval[m], sizeof(T) * kStagedSlots * n)) ||
            (e = cudaMalloc(&plan->pcnt[m], sizeof(int) * n)))
            return e;
        const int g = std::max(1, std::min((P->n + 255) / 256, ctx->num_sms * 16));
        pack_rows_kernel<T><<<g, 256, 0, ctx->stream>>>(P->n, kStagedSlots, M->row, M->col, (const T *)M->val,
                                                        plan->pcol[m], (T *)plan->pval[m], plan->pcnt[m]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) plan->staged_threads = threads;
    return e;
}

static void packed_free(SyncFreePlan *plan)
{
    if (plan->ptiles) cudaFree(plan->ptiles);
    if (plan->far) cudaFree(plan->far);
    if (plan->pack) cudaFree(plan->pack);
    plan->ptiles = nullptr;
    plan->far = nullptr;
    plan->pack = nullptr;
}

static void staged_free(SyncFreePlan *plan)
{
    for (int m = 0; m < 2; ++m) {
        if (plan->pcol[m]) cudaFree(plan->pcol[m]);
        if (plan->pval[m]) cudaFree(plan->pval[m]);
        if (plan->pcnt[m]) cudaFree(plan->pcnt[m]);
        plan->pcol[m] = plan->pcnt[m] = nullptr;
        plan->pval[m] = nullptr;
    }
}

int syncfree_setup(b200la_ctx *ctx, b200la_precond *P)
{
    const char *env = std::getenv("B200LA_SYNCFREE");
    bool use = P->nblocks > 64;
    if (env) use = std::atoi(env) != 0;
    if (!use) return B200LA_OK;
    // Many small levels: one CTA walks them.  Where the operator fits it, on the packed
    // stream; else, with rows of at most four entries, with the cp.async look-ahead
    // (the 7-point 70^3, whose levels of 3,600 rows reach beyond the packed
    // stream's ring, against the register look-ahead: FP64 1,908 -> 1,648 us an apply,
    // FP32 1,681 -> 1,577); else with the register look-ahead.  A variant whose plan
    // finds no memory leaves the operator to the next.
    // (B200LA_SWEEP = staged / lookahead / cta / tickets to start at a variant.)
    const bool few = P->nblocks > 64 && P->n / std::max(P->nblocks, 1) <= 4 * kLevelThreads;
    bool cta = few && P->nblocks <= kLevelMaxLevels, packed = few, staged = few;
    if (const char *sw = std::getenv("B200LA_SWEEP")) {
        packed = std::strcmp(sw, "staged") == 0;
        staged = packed || std::strcmp(sw, "lookahead") == 0;
        cta = (staged || std::strcmp(sw, "cta") == 0) && P->nblocks <= kLevelMaxLevels;
    }
    if (packed || staged || cta) {
        SyncFreePlan *plan = new SyncFreePlan();
        P->syncfree_plan = plan;
        int len = 0, widest = 1;
        for (const b200la_csr *M : {P->L, P->U})
            for (int i = 0; i < M->n; ++i) len = std::max(len, M->h_row[i + 1] - M->h_row[i]);
        for (int l = 0; l < P->nblocks; ++l) widest = std::max(widest, P->block_off[l + 1] - P->block_off[l]);
        cudaError_t e = cudaSuccess;
        auto no_room = [&]() {
            if (e != cudaErrorMemoryAllocation) return;
            cudaGetLastError();
            e = cudaSuccess;
        };
        if (packed && len <= kPackMaxEntries && P->n > 0) {
            e = packed_dispatch(P, len <= 4 ? 4 : len <= 8 ? 8 : 16, [&](auto t, auto kp, auto sgs) {
                return packed_setup<decltype(t), decltype(kp)::value, decltype(sgs)::value>(ctx, P, plan);
            });
            if (!plan->kp) packed_free(plan);
            no_room();
        }
        const int nt = std::min(kLevelThreads, (widest + 31) / 32 * 32);   // idle warps only lengthen a level's barrier
        staged = staged && !plan->kp && len <= kStagedSlots && P->nblocks <= kStagedMaxLevels &&
                 staged_smem<double, kStagedSlots>(P->nblocks, nt) <= kStagedSmemCap;
        if (e == cudaSuccess && !plan->kp && (staged || cta)) {
            plan->nlev = P->nblocks;
            if (!(e = cudaMalloc(&plan->lev_off, sizeof(int) * (P->nblocks + 1))))
                e = setup_copy(ctx->stream, plan->lev_off, P->block_off.data(), sizeof(int) * (P->nblocks + 1));
        }
        if (e == cudaSuccess && staged) {
            e = P->dtype == B200LA_F64 ? staged_setup<double>(ctx, P, plan, nt) : staged_setup<float>(ctx, P, plan, nt);
            if (!plan->staged_threads) staged_free(plan);
            no_room();
        }
        if (e != cudaSuccess) {
            syncfree_free(P);
            return ctx_fail(ctx, B200LA_ERR_ALLOC, "level sweep setup", e);
        }
        if (plan->kp || plan->staged_threads || (cta && plan->lev_off)) {
            P->use_syncfree = 1;
            return B200LA_OK;
        }
        syncfree_free(P);
    }
    const int lgL = lanes_for(P->L), lgU = lanes_for(P->U);
    // chunks of at most 32 >> lg rows, never crossing a block (level) boundary
    auto chunks = [&](int lg, bool reverse) {
        std::vector<int2> out;
        const int per = 32 >> lg;
        for (int k = 0; k < P->nblocks; ++k) {
            const int b = reverse ? P->nblocks - 1 - k : k;
            for (int r = P->block_off[b]; r < P->block_off[b + 1]; r += per)
                out.push_back(make_int2(r, std::min(per, P->block_off[b + 1] - r)));
        }
        return out;
    };
    std::vector<int2> f = chunks(lgL, false), bw = chunks(lgU, true);
    SyncFreePlan *plan = new SyncFreePlan();
    plan->nf = (int)f.size();
    plan->nb = (int)bw.size();
    plan->lg_l = lgL;
    plan->lg_u = lgU;
    cudaError_t e;
    if ((e = cudaMalloc(&plan->fwd, sizeof(int2) * f.size())) || (e = cudaMalloc(&plan->bwd, sizeof(int2) * bw.size())) ||
        (e = setup_copy(ctx->stream, plan->fwd, f.data(), sizeof(int2) * f.size())) ||
        (e = setup_copy(ctx->stream, plan->bwd, bw.data(), sizeof(int2) * bw.size())) ||
        (e = cudaMalloc(&P->flags, sizeof(unsigned) * P->n)) ||
        (e = setup_zero(ctx->stream, P->flags, sizeof(unsigned) * P->n)) ||
        (e = cudaMalloc(&P->sync, sizeof(unsigned) * 4)) ||
        (e = setup_zero(ctx->stream, P->sync, sizeof(unsigned) * 4))) {
        if (plan->fwd) cudaFree(plan->fwd);
        if (plan->bwd) cudaFree(plan->bwd);
        delete plan;
        return ctx_fail(ctx, B200LA_ERR_ALLOC, "syncfree setup", e);
    }
    P->syncfree_plan = plan;
    P->use_syncfree = 1;
    return B200LA_OK;
}

void syncfree_free(b200la_precond *P)
{
    SyncFreePlan *plan = static_cast<SyncFreePlan *>(P->syncfree_plan);
    if (!plan) return;
    if (plan->fwd) cudaFree(plan->fwd);
    if (plan->bwd) cudaFree(plan->bwd);
    if (plan->lev_off) cudaFree(plan->lev_off);
    packed_free(plan);
    staged_free(plan);
    delete plan;
    P->syncfree_plan = nullptr;
}

int syncfree_apply(b200la_ctx *ctx, const b200la_precond *P, const void *r, void *z, const int *gate)
{
    const SyncFreePlan *plan = static_cast<const SyncFreePlan *>(P->syncfree_plan);
    if (plan->kp) {
        PackedSweepArgs a;
        a.tiles = plan->ptiles;
        a.pack = plan->pack;
        a.far = plan->far;
        a.nfar = plan->nfar;
        a.nf = plan->nf_tiles;
        a.nt = plan->nt_tiles;
        a.n = P->n;
        a.stages = plan->stages;
        a.stage_bytes = plan->stage_bytes;
        a.own_off = plan->own_off;
        a.r = r;
        a.z = z;
        a.gate = gate;
        a.err = ctx->dev_err;
        const cudaError_t e = packed_dispatch(P, plan->kp, [&](auto t, auto kp, auto sgs) {
            return packed_launch<decltype(t), decltype(kp)::value, decltype(sgs)::value>(plan, a, ctx->stream);
        });
        if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "packed level sweep", e);
        ctx->launches += 1;
        return B200LA_OK;
    }
    if (plan->staged_threads) {
        LevelStagedArgs a;
        a.off = plan->lev_off;
        a.nlev = plan->nlev;
        a.n = P->n;
        a.r = r;
        a.z = z;
        a.d1 = P->iDv;
        a.d2 = P->Dv;
        a.sgs = P->kind == B200LA_PRECOND_MCSGS;
        a.gate = gate;
        for (int dir = 0; dir < 2; ++dir) {
            a.pcol = plan->pcol[dir];
            a.pval = plan->pval[dir];
            a.pcnt = plan->pcnt[dir];
            a.backward = dir;
            const int nt = plan->staged_threads;
            if (P->dtype == B200LA_F64)
                level_sweep_staged_kernel<double, kStagedSlots>
                    <<<1, nt, staged_smem<double, kStagedSlots>(plan->nlev, nt), ctx->stream>>>(a);
            else
                level_sweep_staged_kernel<float, kStagedSlots>
                    <<<1, nt, staged_smem<float, kStagedSlots>(plan->nlev, nt), ctx->stream>>>(a);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "staged level sweep", e);
            ctx->launches += 1;
        }
        return B200LA_OK;
    }
    if (plan->lev_off) {
        LevelSweepArgs a;
        a.off = plan->lev_off;
        a.nlev = plan->nlev;
        a.r = r;
        a.z = z;
        a.d1 = P->iDv;
        a.d2 = P->Dv;
        a.sgs = P->kind == B200LA_PRECOND_MCSGS;
        a.gate = gate;
        for (int dir = 0; dir < 2; ++dir) {
            const b200la_csr *M = dir ? P->U : P->L;
            a.row = M->row;
            a.col = M->col;
            a.val = M->val;
            a.backward = dir;
            if (P->dtype == B200LA_F64)
                level_sweep_cta_kernel<double>
                    <<<1, kLevelThreads, kLevelRing * sizeof(double) + sizeof(int) * (plan->nlev + 1), ctx->stream>>>(a);
            else
                level_sweep_cta_kernel<float>
                    <<<1, kLevelThreads, kLevelRing * sizeof(float) + sizeof(int) * (plan->nlev + 1), ctx->stream>>>(a);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "level sweep", e);
            ctx->launches += 1;
        }
        return B200LA_OK;
    }
    SyncFreeArgs a;
    a.r = r;
    a.z = z;
    a.d1 = P->iDv;
    a.d2 = P->Dv;
    a.flags = P->flags;
    a.sync = P->sync;
    a.sgs = P->kind == B200LA_PRECOND_MCSGS;
    a.gate = gate;
    a.err = ctx->dev_err;
    const int grid = ctx->num_sms * 4;
    for (int dir = 0; dir < 2; ++dir) {
        const b200la_csr *M = dir ? P->U : P->L;
        a.row = M->row;
        a.col = M->col;
        a.val = M->val;
        a.chunks = dir ? plan->bwd : plan->fwd;
        a.nchunks = dir ? plan->nb : plan->nf;
        a.lg = dir ? plan->lg_u : plan->lg_l;
        a.backward = dir;
        if (P->dtype == B200LA_F64)
            syncfree_sweep_kernel<double><<<grid, kBlock, 0, ctx->stream>>>(a);
        else
            syncfree_sweep_kernel<float><<<grid, kBlock, 0, ctx->stream>>>(a);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return ctx_fail(ctx, B200LA_ERR_CUDA, "syncfree sweep", e);
        ctx->launches += 1;
    }
    return B200LA_OK;
}
