// fd3d_selftest.cu -- checks that run on the device: the PML quotients against the IEEE division,
// over every dividend, and the bounded waits.
//
// The PML updates divide by dh and by 1 + omega, divisors known before the launch; div_by and
// div_by_signed (fd3d_common.cuh) form those quotients from a pair made on the host, div_steps
// those of a divisor without one, and div_small and div_exact those they do not cover.
// fd3d_check_division runs them, chosen as the sweeps choose them, and __fdiv_rn on every one of the
// 2^32 float bit patterns for each divisor given and counts the dividends whose results differ in
// any bit (two NaNs count as equal).
#include <cuda_runtime.h>
#include <cstdint>
#include "../../include/fd3d_gpu.h"
#include "fd3d_common.cuh"
#include "fd3d_setup.h"

using namespace fd3d;

namespace {

struct Pair { float h, l, s; int ok; };

// as quotient() below, for PML_STEPS: y = RN(1/b)
__device__ float quotient_steps(float x, float b, float y, float s) {
    unsigned key = 0xffffffffu;
    const float q = div_steps(x * s, b, y, key) * (1.0f / s);
    if (!pml_finite(q)) return div_exact(x, b);
    return key < DIV_KEY ? div_small<true>(x, b, y, 0.0f) : q;
}

// the sweeps' quotient: div_by on the scaled dividend, or what its key or result asks for
__device__ float quotient(float x, float b, const Pair& y, bool sign) {
    unsigned key = 0xffffffffu;
    const float xs = x * y.s, q = (sign ? div_by_signed(xs, y.h, y.l, key) : div_by(xs, y.h, y.l, key)) * (1.0f / y.s);
    if (!y.ok || !pml_finite(q)) return div_exact(x, b);
    return key < DIV_KEY ? div_small<false>(x, b, y.h, y.l) : q;
}

// y: the pair with l >= 0 (the divisor dh), ys: the pair of any sign (1 + omega), recip: RN(1/b), 0
// for a divisor out of range
__global__ void k_check_division(float b, Pair y, Pair ys, float recip, unsigned long long* bad, unsigned* first) {
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long local = 0;
    unsigned ex = 0;
    for (uint64_t n = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; n < (1ull << 32); n += nthreads) {
        const unsigned bits = (unsigned)n;
        const float x = __uint_as_float(bits);
        const float r = __fdiv_rn(x, b);
        auto is = [&](float q) { return (__float_as_uint(q) == __float_as_uint(r)) || (q != q && r != r); };
        bool same = is(quotient(x, b, y, false)) && is(quotient(x, b, ys, true)) && is(div_exact(x, b));
        if (ys.ok && pml_finite(x)) same = same && is(div_small<false>(x, b, ys.h, ys.l));
        if (recip != 0.0f) same = same && is(quotient_steps(x, b, recip, y.s)) && (!pml_finite(r) || is(div_small<true>(x, b, recip, 0.0f)));
        if (!same) {
            if (local == 0) ex = bits;
            ++local;
        }
    }
    if (local) {
        atomicAdd(bad, local);
        atomicCAS(first, 0xffffffffu, ex);
    }
}

// ---------------------------------------------------------------- self-test of the waits
// An mbarrier phase that no copy or arrival completes, and a grid barrier that one CTA
// never reaches: both waits must give up by their bound, record ST_TIMEOUT and return,
// leaving the context usable (failure detection without a hung or faulted GPU).
__global__ void k_check_mbar_wait(int* status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) { mbar_init(smem_addr(&bar), 1); fence_mbar_init(); }
    __syncthreads();
    const bool done = mbar_wait(smem_addr(&bar), 0u);  // nothing ever arrives on this phase
    if (__syncthreads_or(!done) && threadIdx.x == 0) atomicOr(status, ST_TIMEOUT);
}

struct BarrierSync {
    unsigned count;
    unsigned gen;
    int abort;
    int pad;
};

constexpr int BARRIER_SPIN_LIMIT = 1 << 22;

// Sense-counting grid barrier with a bounded spin; false if this CTA gave up (or another did).  No
// kernel of a step waits for another CTA: this is the pattern of such a wait, kept under test.
__device__ bool grid_barrier(BarrierSync* b, unsigned nblocks, int* status) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        ok = 1;
        volatile unsigned* vgen = &b->gen;
        volatile int* vab = &b->abort;
        const unsigned g0 = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(&b->count, 1u);
        if (arrived == nblocks - 1) {
            atomicExch(&b->count, 0u);
            __threadfence();
            atomicAdd(&b->gen, 1u);
        } else {
            int n = 0;
            while (*vgen == g0) {
                if (*vab) { ok = 0; break; }
                if (++n > BARRIER_SPIN_LIMIT) {
                    atomicOr(status, ST_TIMEOUT);
                    atomicExch(&b->abort, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

__global__ void k_check_grid_barrier(BarrierSync* sync, int* status) {
    if (blockIdx.x == gridDim.x - 1) return;  // this CTA never arrives
    grid_barrier(sync, gridDim.x, status);
}

}  // namespace

static_assert(FD3D_DIVISION_PAIR == PML_PAIR && FD3D_DIVISION_SIGNED == PML_SIGNED && FD3D_DIVISION_STEPS == PML_STEPS &&
              FD3D_DIVISION_EXACT == PML_EXACT, "the header's forms are PmlForm's");
extern "C" int fd3d_division_form(float divisor, int damping, int* form) {
    if (!form) return FD3D_ERR_ARG;
    float h, l, y;
    *form = div_form(divisor, damping != 0, h, l, y);
    return FD3D_OK;
}

extern "C" int fd3d_check_division(const float* divisors, int n, unsigned long long* mismatches,
                                   unsigned* first_bad) {
    if (!divisors || n < 0 || !mismatches) return FD3D_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return FD3D_ERR_NODEV; }
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FD3D_ERR_CUDA;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return FD3D_ERR_CUDA;
    unsigned long long* dbad = nullptr;
    unsigned* dfirst = nullptr;
    if (cudaMalloc(&dbad, sizeof(unsigned long long)) != cudaSuccess) return FD3D_ERR_NOMEM;
    if (cudaMalloc(&dfirst, sizeof(unsigned)) != cudaSuccess) { cudaFree(dbad); return FD3D_ERR_NOMEM; }
    int rc = FD3D_OK;
    for (int i = 0; i < n && rc == FD3D_OK; ++i) {
        const float b = divisors[i];
        Pair y, ys;
        y.s = ys.s = b > 0 ? (float)div_scale(b) : 1.0f;
        y.ok = div_pair(b, true, y.h, y.l);
        ys.ok = div_pair(b, false, ys.h, ys.l);
        const float recip = div_in_range(b) ? ys.h : 0.0f;
        const unsigned none = 0xffffffffu;
        if (cudaMemset(dbad, 0, sizeof(unsigned long long)) != cudaSuccess ||
            cudaMemcpy(dfirst, &none, sizeof(unsigned), cudaMemcpyHostToDevice) != cudaSuccess) {
            rc = FD3D_ERR_CUDA;
            break;
        }
        k_check_division<<<nsm * 8, 256>>>(b, y, ys, recip, dbad, dfirst);
        unsigned long long hb = 0;
        unsigned hf = none;
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
            cudaMemcpy(&hb, dbad, sizeof(hb), cudaMemcpyDeviceToHost) != cudaSuccess ||
            cudaMemcpy(&hf, dfirst, sizeof(hf), cudaMemcpyDeviceToHost) != cudaSuccess) {
            rc = FD3D_ERR_CUDA;
            break;
        }
        mismatches[i] = hb;
        if (first_bad) first_bad[i] = hf;
    }
    cudaFree(dbad);
    cudaFree(dfirst);
    return rc;
}

extern "C" int fd3d_check_waits(int* mbar_status, int* barrier_status) {
    if (!mbar_status || !barrier_status) return FD3D_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return FD3D_ERR_NODEV; }
    int* st = nullptr;
    BarrierSync* sync = nullptr;
    if (cudaMalloc(&st, 2 * sizeof(int)) != cudaSuccess) return FD3D_ERR_NOMEM;
    if (cudaMalloc(&sync, sizeof(BarrierSync)) != cudaSuccess) { cudaFree(st); return FD3D_ERR_NOMEM; }
    int rc = FD3D_OK, h[2] = {0, 0};
    if (cudaMemset(st, 0, 2 * sizeof(int)) != cudaSuccess || cudaMemset(sync, 0, sizeof(BarrierSync)) != cudaSuccess)
        rc = FD3D_ERR_CUDA;
    if (rc == FD3D_OK) {
        k_check_mbar_wait<<<1, 64>>>(st);
        k_check_grid_barrier<<<2, 64>>>(sync, st + 1);
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
            cudaMemcpy(h, st, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
            rc = FD3D_ERR_CUDA;
    }
    cudaFree(st);
    cudaFree(sync);
    *mbar_status = h[0];
    *barrier_status = h[1];
    return rc;
}
