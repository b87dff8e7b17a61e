// grid_gather.cuh -- sums over the whole grid inside one cooperative launch.
//
// A solver step whose vectors fit the chip spends its time on launches and
// reduction tails, not on bytes.  Here every CTA writes its partial sum and the
// epoch of the sum as one 16-byte word, and every CTA polls the words of all
// CTAs until they carry that epoch: one trip through L2 stands between a partial
// and its total, no atomic and no fence, where a kernel boundary costs several
// microseconds.  All CTAs add the partials in the same order, so they hold the
// same bits and take the same decisions.  A CTA's words have a line of their own.
// Per iteration of a CG with two sums and 130 CTAs, in one call: 7.0 us; 4 to 32 copies
// of the words 7.8, a mailbox per reader 7.5, a CTA that collects and hands out the
// total (two trips) 8.6, words published and polled with release and acquire 12.7.
// In another: 8.1 us, and 11.0 with the words of four CTAs on a line.
//
// Epochs rise through the life of the context.  Words are double-buffered by
// the epoch's parity: a CTA writes epoch k + 2 only after it has seen k + 1 of
// every CTA, which each writes after it has read k.  Polls are bounded; after
// one has run out (reported in the error flag) nothing waits any more, nor in a
// later launch until the host has seen the flag.  A sum that lacks a word is
// infinite, which ends a solve by its own stop test.  (A test for it in the CG's
// loop took 0.1 us of a small iteration's 3.1 and made the streaming form spill:
// 80^3 FP64 25.1 -> 27.8 us.)  The CTAs' epochs may differ then, so the host clears
// the words and the saved epoch with the flag (ctx_check_device_error): a word
// never carries an epoch to come.
#pragma once

#include <algorithm>
#include <cstdlib>

#include "common.cuh"

namespace b200 {

constexpr int kGatherMaxQ = 2;         // quantities per sum
constexpr int kGatherMaxCtas = 160;    // CTAs of a gathering grid
constexpr long long kGatherSpin = 1LL << 22;   // polls of one wait: several seconds
constexpr size_t kGatherBytes = 128 * (1 + (size_t)2 * kGatherMaxCtas);   // the last epoch, the words of two epochs

// CTAs that a gathering grid may have: one per SM.  (B200LA_GATHER_CTAS: another number.
// Where they are not all resident at once the launch is refused and the solvers
// take a launch per step.)
inline int gather_ctas(int num_sms)
{
    const char *e = std::getenv("B200LA_GATHER_CTAS");
    return std::max(1, std::min(e ? std::atoi(e) : num_sms, kGatherMaxCtas));
}

// B200LA_GATHER_SPIN: polls after which a wait gives up (-1: at the first word that is not there yet)
// -- as the number of the first poll, counted up to kGatherSpin.
inline int gather_first()
{
    const char *e = std::getenv("B200LA_GATHER_SPIN");
    return e ? (int)(kGatherSpin - std::min(std::max(std::atoll(e), -1LL), kGatherSpin)) : 0;
}

__device__ __forceinline__ void st_word(void *p, double v, unsigned long long e)
{
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(e) : "memory");
}
__device__ __forceinline__ void ld_word(const void *p, double &v, unsigned long long &e)
{
    long long x;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(x), "=l"(e) : "l"(p) : "memory");
    v = __longlong_as_double(x);
}

// One per kernel; all threads of all CTAs construct it and call its members
// together.  THREADS: threads of a CTA (at least kGatherMaxCtas).
template <int THREADS>
struct GridGather {
    static_assert(THREADS >= kGatherMaxCtas, "one thread per CTA's word");
    struct Shared {
        double part[kGatherMaxQ][THREADS / 32], tot[kGatherMaxQ][kGatherMaxCtas / 32];
        int fail;
    };
    unsigned char *words;
    unsigned long long epoch;
    Shared &sh;
    int *err;
    const int first;   // number of a wait's first poll

    // `mem`: kGatherBytes of the context (the last epoch used, then the words)
    __device__ GridGather(unsigned char *mem, Shared &s, int *e, int f)
        : words(mem + 128), sh(s), err(e), first(f)
    {
        epoch = __ldcg(reinterpret_cast<const unsigned long long *>(mem));
        if (threadIdx.x == 0) sh.fail = __ldcg(e) != kDevOk;
        __syncthreads();
    }
    // after the last sum, by CTA 0: the next kernel goes on from there
    __device__ void close()
    {
        if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned long long *>(words - 128) = epoch;
    }
    // After the last wait: whether one of this CTA's has run out (or the flag was up before), in all threads.
    __device__ bool failed()
    {
        __syncthreads();
        return *static_cast<volatile int *>(&sh.fail) != 0;
    }
    // Publish this CTA's sums of v.  (Nothing else is ordered by it: data that
    // CTAs exchange carry epochs themselves, as a fence costs about 1 us.)
    template <int NQ>
    __device__ void publish(const double (&v)[NQ])
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double w = warp_sum(v[q]);
            if (lane == 0) sh.part[q][warp] = w;
        }
        __syncthreads();
        ++epoch;
        if (warp == 0) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double s = warp_sum(lane < THREADS / 32 ? sh.part[q][lane] : 0.0);
                if (lane == q) st_word(word(blockIdx.x, q), s, epoch);
            }
        }
    }
    // Totals of the sums published last, in every thread.
    template <int NQ>
    __device__ void total(double (&out)[NQ])
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ctas = gridDim.x;
        if (warp * 32 < ctas) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double w = warp_sum((int)threadIdx.x < ctas ? poll(word(threadIdx.x, q)) : 0.0);
                if (lane == 0) sh.tot[q][warp] = w;
            }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            double s = 0.0;
            for (int w = 0; w * 32 < ctas; ++w) s += sh.tot[q][w];
            out[q] = s;
        }
    }
    // All CTAs meet, and what their threads wrote before may be read after.
    __device__ void sync()
    {
        __syncthreads();
        ++epoch;
        if (threadIdx.x == 0) {
            fence();
            st_word(word(blockIdx.x, 0), 0.0, epoch);
        }
        if ((int)(threadIdx.x & ~31u) < (int)gridDim.x) {
            if (threadIdx.x < gridDim.x) poll(word(threadIdx.x, 0));
            __syncwarp();
            fence();
        }
        __syncthreads();
    }
    // after an unsuccessful poll number i: true when to give up
    __device__ bool stop(long long i)
    {
        volatile int *fail = &sh.fail;
        if (*fail) return true;
        if (i > kGatherSpin) {
            *fail = 1;
            atomicExch(err, kDevWaitTimeout);
        }
        return false;
    }

private:
    __device__ static void fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
    __device__ double poll(const void *p)
    {
        double v;
        unsigned long long e;
        ld_word(p, v, e);
        for (long long i = first; e != epoch; ++i) {
            if (stop(i)) return __longlong_as_double(0x7ff0000000000000LL);
            ld_word(p, v, e);
        }
        return v;
    }
    __device__ void *word(int cta, int q)
    {
        return words + 128 * ((int)(epoch & 1) * kGatherMaxCtas + cta) + 16 * q;
    }
};

}  // namespace b200
