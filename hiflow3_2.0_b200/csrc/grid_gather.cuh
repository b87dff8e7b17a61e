// grid_gather.cuh -- sums over the whole grid inside one cooperative launch.
//
// A solver step whose vectors fit the chip spends its time on launches and
// reduction tails, not on bytes.  Here every CTA publishes its partial sum and
// the epoch of the sum as one 16-byte word, and every CTA polls the words of
// all CTAs until they carry that epoch: one L2 write and one L2 read stand
// between a partial and its total (about 1 us over 148 CTAs), where a ticket
// barrier takes an atomic, a flag and the read of the partials behind it, and
// a kernel boundary several microseconds.  All CTAs add the partials in the
// same order, so they hold the same bits and take the same decisions.
//
// Epochs rise through the life of the context.  Words are double-buffered by
// the epoch's parity: a CTA publishes epoch k + 2 only after every CTA has
// published k + 1, which each does after it has read k.  Polls are bounded;
// after one has run out (reported in the error flag) nothing waits any more.
#pragma once

#include "common.cuh"

namespace b200 {

constexpr int kGatherMaxQ = 2;         // quantities per sum
constexpr int kGatherMaxCtas = 160;    // CTAs of a gathering grid
constexpr long long kGatherSpin = 1LL << 22;
constexpr size_t kGatherBytes = 16 + 16 * (size_t)2 * kGatherMaxQ * kGatherMaxCtas;

__device__ __forceinline__ void st_word(void *p, double v, unsigned long long e, bool release)
{
    if (release)
        asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.release.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                     "l"(__double_as_longlong(v)), "l"(e) : "memory");
    else
        asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                     "l"(__double_as_longlong(v)), "l"(e) : "memory");
}
__device__ __forceinline__ void ld_word(const void *p, double &v, unsigned long long &e, bool acquire)
{
    long long x;
    if (acquire)
        asm volatile("{\n\t.reg .b128 w;\n\tld.acquire.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                     : "=l"(x), "=l"(e) : "l"(p) : "memory");
    else
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

    // `mem`: kGatherBytes of the context (the last epoch used, then the words)
    __device__ GridGather(unsigned char *mem, Shared &s, int *e) : words(mem + 16), sh(s), err(e)
    {
        epoch = __ldcg(reinterpret_cast<const unsigned long long *>(mem));
        if (threadIdx.x == 0) sh.fail = 0;
        __syncthreads();
    }
    // after the last sum, by CTA 0: the next kernel goes on from there
    __device__ void close()
    {
        if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned long long *>(words - 16) = epoch;
    }
    // Publish this CTA's sums of v (ORDERED: with everything its threads wrote before).
    template <int NQ, bool ORDERED>
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
                if (lane == q) st_word(word(q, blockIdx.x), s, epoch, ORDERED);
            }
        }
    }
    // Totals of the sums published last, in every thread (ORDERED: what the
    // CTAs wrote before publishing may be read).
    template <int NQ, bool ORDERED>
    __device__ void total(double (&out)[NQ])
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ctas = gridDim.x;
        double v[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = 0.0;
        if ((int)threadIdx.x < ctas) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                unsigned long long e;
                volatile int *fail = &sh.fail;
                ld_word(word(q, threadIdx.x), v[q], e, ORDERED);
                for (long long i = 0; e != epoch && !*fail; ++i) {
                    if (i > kGatherSpin) {
                        *fail = 1;
                        atomicExch(err, kDevWaitTimeout);
                    }
                    ld_word(word(q, threadIdx.x), v[q], e, ORDERED);
                }
            }
        }
        if (warp * 32 < ctas) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const double w = warp_sum(v[q]);
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

private:
    __device__ void *word(int q, int cta)
    {
        return words + 16 * (((epoch & 1) * kGatherMaxQ + q) * kGatherMaxCtas + cta);
    }
};

}  // namespace b200
