// Device helpers shared by the kernel files of the phx library (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "phx_internal.h"

namespace phx {

static constexpr int kThreads = 256;

template <class T> __device__ __forceinline__ T ld(const T *p) { return __ldg(p); }
// Loads of data written earlier in the same kernel by other blocks: bypass L1.
template <class T> __device__ __forceinline__ T ldcg(const T *p) { return __ldcg(p); }

// Vector loads of 4- or 8-element records (16-byte aligned).
__device__ __forceinline__ void ld4(const double *p, double *o)
{
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ void ld4(const float *p, float *o)
{
    const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
}
template <class T>
__device__ __forceinline__ void ld8(const T *p, T *o) { ld4(p, o); ld4(p + 4, o + 4); }
__device__ __forceinline__ void st4(double *p, const double *v)
{
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void st4(float *p, const float *v)
{
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
}
template <class T>
__device__ __forceinline__ void st8(T *p, const T *v) { st4(p, v); st4(p + 4, v + 4); }

// Writes state, c2 = |gamma p / rho| and total enthalpy of a cell record
// (slot 7, the limiter, is left untouched).  c2 and the enthalpy are the
// per-cell factors MXDQ_STD forms (Jacobian.cpp:22-23, PerfectGas.cpp:384-394).
template <class T>
__device__ __forceinline__ void put_state(T *rec, const T *q, T gm)
{
    const T c2 = fabs(gm * q[4] / q[0]);
    const T hm = (gm / (gm - T(1))) * (q[4] / q[0]) + T(0.5) * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    T v[4] = {q[0], q[1], q[2], q[3]};
    st4(rec, v);
    rec[4] = q[4];
    rec[5] = c2;
    rec[6] = hm;
}

// Temperature (ComputeGamaAndTemperature, NSSolverUnstruct.cpp:4717-4730) and
// Sutherland viscosity (ComputeViscousCoefficientWithoutChemical, :6722-6747),
// formed on the fly from a cell record wherever they are needed.
template <class T>
__device__ __forceinline__ T temperature(const T *q, T coef) { return q[4] / (coef * q[0]); }
template <class T>
__device__ __forceinline__ T sutherland(T t, T s) { return t * sqrt(t) * (T(1) + s) / (t + s); }

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
}

// Bounded wait for the mbarrier phase with the given parity; false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity)
{
    const uint32_t a = smem_u32(mbar);
    for (long long i = 0; i < (1LL << 26); ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void mbar_expect(uint64_t *mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes) : "memory");
}

// Bulk copy of global memory into shared memory (addresses and size multiples of
// 16 bytes) of data read once: it leaves L2 first.
__device__ __forceinline__ uint64_t evict_first_policy()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *mbar, uint64_t policy)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(mbar)), "l"(policy)
        : "memory");
}

// IEEE division on both paths, for the LU-SGS sweeps: the files holding the
// face and SA passes are compiled with approximate FP32 division.
__device__ __forceinline__ float idiv(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double idiv(double a, double b) { return a / b; }

// A row of the LU-SGS schedule is one warp: kSweepLanes lanes a cell.
static_assert(kSweepLanes * kSweepSlots == 32, "one warp holds kSweepSlots slots");

// The rows of one warp on their way through its shared memory: two rows of
// kRow bytes a stage, `stages` stages, each filled by one bulk copy (a warp's
// rows are contiguous) that lane 0 issues.  Gathered lane by lane instead, the
// copies' address arithmetic took more instructions than the row's own work,
// and one warp issues them one after the other.
template <int kRow>
struct RowPipe {
    static constexpr int kStage = 2 * kRow;
    unsigned char *buf;
    uint64_t *full;
    const unsigned char *src;         // the warp's next stage to be issued
    int nrow, nstage, stages;         // rows, stages of rows, stages in flight
    int slot, ahead;                  // slot of the current stage; stages issued
    uint32_t parity;
    uint64_t policy;

    __device__ __forceinline__ unsigned char *at(int sl) const { return buf + sl * kStage; }
    __device__ __forceinline__ void issue(int sl, int lane)
    {
        if (lane == 0) {
            const uint32_t n = (uint32_t)min(2, nrow - 2 * ahead) * kRow;
            mbar_expect(full + sl, n);
            bulk_load(at(sl), src, n, full + sl, policy);
        }
        src += kStage;
        ++ahead;
    }
    __device__ __forceinline__ void start(unsigned char *mem, uint64_t *bars, const unsigned char *rows, int row0, int n,
                                          int st, int lane)
    {
        buf = mem;
        full = bars;
        src = rows + (size_t)row0 * kRow;
        nrow = n;
        nstage = (n + 1) / 2;
        stages = st;
        slot = ahead = 0;
        parity = 0;
        policy = evict_first_policy();
        if (lane == 0) {
            for (int i = 0; i < st; ++i) mbar_init(full + i, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int i = 0; i < st && i < nstage; ++i) issue(i, lane);
        __syncwarp();
    }
    __device__ __forceinline__ bool wait() const { return mbar_wait(full + slot, parity); }
    // after all lanes have read the current stage
    __device__ __forceinline__ void advance(int lane)
    {
        if (ahead < nstage) issue(slot, lane);
        if (++slot == stages) { slot = 0; parity ^= 1u; }
    }
    // before leaving early at stage k: the copies in flight
    __device__ __forceinline__ void drain(int k) const
    {
        int sl = slot;
        uint32_t p = parity;
        for (; k < ahead; ++k) {
            mbar_wait(full + sl, p);
            if (++sl == stages) { sl = 0; p ^= 1u; }
        }
    }
};

// Factors of one face use (kUse values), in 16-byte units rotated by the lane so
// that a warp reads them from shared memory without bank conflicts.
__device__ __forceinline__ void put_use(float *use, int lane, const float *v)
{
    const int x = (lane >> 2) & 1;
    st4(use + 4 * x, v);
    st4(use + 4 * (1 - x), v + 4);
}
__device__ __forceinline__ void put_use(double *use, int lane, const double *v)
{
#pragma unroll
    for (int k = 0; k < 4; ++k)
        reinterpret_cast<double2 *>(use)[(k + (lane >> 1)) & 3] = make_double2(v[2 * k], v[2 * k + 1]);
}
__device__ __forceinline__ void get_use(const float *use, int lane, float *v)
{
    const int x = (lane >> 2) & 1;
    const float4 a = reinterpret_cast<const float4 *>(use)[x], b = reinterpret_cast<const float4 *>(use)[1 - x];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void get_use(const double *use, int lane, double *v)
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double2 a = reinterpret_cast<const double2 *>(use)[(k + (lane >> 1)) & 3];
        v[2 * k] = a.x; v[2 * k + 1] = a.y;
    }
}
// 4 or 8 values of shared memory
__device__ __forceinline__ void get4(const float *p, float *o)
{
    const float4 a = *reinterpret_cast<const float4 *>(p);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
}
__device__ __forceinline__ void get4(const double *p, double *o)
{
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
template <class T>
__device__ __forceinline__ void get8(const T *p, T *o) { get4(p, o); get4(p + 4, o + 4); }

// Write-once sweep records.  Before a sweep every element of its output
// records holds the sentinel, a NaN whose sign and payload no arithmetic
// result carries: single-precision arithmetic gives no NaN but the positive
// canonical one, and in double precision, which may hand a NaN operand on,
// producers map the sentinel pattern to another NaN.  During the sweep
// each element is stored once, so a reader that sees anything but the
// sentinel sees the final value: the data is its own completion flag, and
// neither a fence between the producer's stores nor a second load after the
// wait sits on the sweep's critical path.  Stores and polling loads are
// relaxed at device scope (coherent in L2, not cached in L1).
static constexpr unsigned kSentinelF = 0xffc0e1a5u;
static constexpr unsigned long long kSentinelD = 0xfff80000d0e1a5c3ull;

template <class T> __device__ __forceinline__ T sweep_sentinel();
template <> __device__ __forceinline__ float sweep_sentinel<float>() { return __uint_as_float(kSentinelF); }
template <> __device__ __forceinline__ double sweep_sentinel<double>()
{
    return __longlong_as_double((long long)kSentinelD);
}
__device__ __forceinline__ bool is_sentinel(float v) { return __float_as_uint(v) == kSentinelF; }
__device__ __forceinline__ bool is_sentinel(double v)
{
    return (unsigned long long)__double_as_longlong(v) == kSentinelD;
}
// a computed value as stored
__device__ __forceinline__ float unsentinel(float v) { return v; }
__device__ __forceinline__ double unsentinel(double v)
{
    return is_sentinel(v) ? __longlong_as_double(0x7fffffffffffffffLL) : v;
}

__device__ __forceinline__ float ld_poll(const float *p)
{
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_poll(const double *p)
{
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(float *p, float v)
{
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(double *p, double v)
{
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// Polls the first five elements of an 8-element record: the loads alone (the
// values are looked at later), whether none of them is the sentinel (they are
// then final), and both together.
__device__ __forceinline__ void poll5_load(const float *p, float *o)
{
    asm volatile(
        "{\n\t.reg .f32 x, y, z;\n\t"
        "ld.relaxed.gpu.global.v8.f32 {%0, %1, %2, %3, %4, x, y, z}, [%5];\n\t}\n"
        : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4])
        : "l"(p)
        : "memory");
}
__device__ __forceinline__ void poll5_load(const double *p, double *o)
{
    asm volatile("ld.relaxed.gpu.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
                 : "l"(p)
                 : "memory");
    o[4] = ld_poll(p + 4);
}
template <class T>
__device__ __forceinline__ bool poll5_done(const T *o)
{
    return !(is_sentinel(o[0]) | is_sentinel(o[1]) | is_sentinel(o[2]) | is_sentinel(o[3]) | is_sentinel(o[4]));
}
template <class T>
__device__ __forceinline__ bool poll5(const T *p, T *o)
{
    poll5_load(p, o);
    return poll5_done(o);
}

// Publishes the five values of an 8-element record (the rest zero): whole
// sectors, so that L2 need not fetch the sentinel's from DRAM to complete them.
__device__ __forceinline__ void publish5(float *p, const float *v)
{
    asm volatile("st.relaxed.gpu.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %6, %6};" ::"l"(p), "f"(unsentinel(v[0])),
                 "f"(unsentinel(v[1])), "f"(unsentinel(v[2])), "f"(unsentinel(v[3])), "f"(unsentinel(v[4])), "f"(0.0f)
                 : "memory");
}
__device__ __forceinline__ void publish5(double *p, const double *v)
{
    asm volatile("st.relaxed.gpu.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(unsentinel(v[0])),
                 "d"(unsentinel(v[1])), "d"(unsentinel(v[2])), "d"(unsentinel(v[3]))
                 : "memory");
    asm volatile("st.relaxed.gpu.global.v4.f64 [%0], {%1, %2, %2, %2};" ::"l"(p + 4), "d"(unsentinel(v[4])), "d"(0.0)
                 : "memory");
}

}  // namespace phx
