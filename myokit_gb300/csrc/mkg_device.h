/*
 * mkg_device.h -- waits shared by the generated kernels, prepended as text.
 */
static __device__ __forceinline__ unsigned long long mkg_clock_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

static __device__ __forceinline__ unsigned int mkg_ld_acquire(
    const unsigned int *p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];"
                 : "=r"(v) : "l"(p) : "memory");
    return v;
}

static __device__ __forceinline__ int mkg_ld_volatile_int(const int *p)
{
    return *((const volatile int *)p);
}

// Publishes a step counter: what this thread wrote (and saw) before is
// visible to a thread that acquires it
static __device__ __forceinline__ void mkg_st_release(unsigned int *p,
                                                      unsigned int v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;"
                 :: "l"(p), "r"(v) : "memory");
}

// Grid-wide barrier over a co-resident (cooperative) grid. Every block
// arrives once per barrier, so barrier number e completes when the low 31
// bits of the counter reach e * gridDim (the host keeps that below 2^31).
// The wait gives up after timeout_ns (or as soon as another block reported
// an error), records MKG_DEV_TIMEOUT and returns false; the caller then
// leaves the kernel, so no wait is ever unbounded. It also returns false,
// in every block, after a NaN halt at or before step halt_at (see below).
#define MKG_HALT_BIT 0x80000000u
static __device__ __forceinline__ bool mkg_grid_barrier(
    mkg_status *st, unsigned int epoch, long long timeout_ns, int *s_ok,
    int halt_at = -1)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int target = epoch * gridDim.x;
        // A NaN halt recorded at or before step halt_at (by this CTA's
        // threads, ordered before this by the CTA barrier) sets the
        // counter's top bit before this CTA arrives
        if (halt_at >= 0 && mkg_ld_volatile_int(&st->halt_step) <= halt_at)
            asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;"
                         :: "l"(&st->barrier), "r"(MKG_HALT_BIT)
                         : "memory");
        // Release: the CTA's writes, ordered before this by the CTA
        // barrier, are visible to every block that acquires the count
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;"
                     :: "l"(&st->barrier) : "memory");
        int ok = 1;
        unsigned int c = mkg_ld_acquire(&st->barrier);
        if ((c & ~MKG_HALT_BIT) < target) {
            const unsigned long long t0 = mkg_clock_ns();
            while (((c = mkg_ld_acquire(&st->barrier)) & ~MKG_HALT_BIT) <
                   target) {
                if (mkg_ld_volatile_int(&st->error) != MKG_DEV_OK) {
                    ok = 0;
                    break;
                }
                if ((long long)(mkg_clock_ns() - t0) > timeout_ns) {
                    atomicCAS(&st->error, MKG_DEV_OK, MKG_DEV_TIMEOUT);
                    atomicExch(&st->timeout_block, (int)blockIdx.x);
                    ok = 0;
                    break;
                }
                __nanosleep(32);
            }
        }
        // Every block leaves after a barrier that completed with the halt
        // bit set (the counter is reset per chunk)
        if (c & MKG_HALT_BIT) ok = 0;
        // The acquire loads order what the CTA reads after the barrier
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}
