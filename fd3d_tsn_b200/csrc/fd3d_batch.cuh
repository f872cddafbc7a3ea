// fd3d_batch.cuh -- the batch's work items, its models' descriptors, and the kernels that hold PML
// tiles (fd3d_batch.cu has those whose quotients are PML_PAIR, fd3d_forms.cu the others).
#pragma once
#include "fd3d_common.cuh"
#include "fd3d_kernels.cuh"
#include "fd3d_opt.cuh"

namespace fd3d {

enum WorkType : int {
    W_VEL_INT = 0, W_VEL_FAULT, W_VEL_PML, W_VEL_FS, W_STR_INT, W_STR_FAULT, W_STR_PML, W_STR_FS, W_FBC, W_NUC
};
struct Work {
    int tm;          // type | model << 8
    int bx, by, bz;
};

// what the sweeps read of a model: a CTA copies it to shared memory first (load_par), where a
// store to the wave field cannot alias it (from global memory each pointer and size was
// loaded again after each store: 705 instructions a cell in the stress PML tiles)
struct ModelPar {
    Grid g;
    Fields<float> f;
    StepConst<float> c;
    PmlDesc D;
    PmlAux<float> X;
};

struct ModelDev : ModelPar {
    Fault<float> q;
    FvwScalars fs;
    HistDesc h;
    int law;
    int* it_dev;
    int* status;
    double* psiX0;
    double* psiZ0;
};

// every thread of the CTA calls it
__device__ __forceinline__ void load_par(ModelPar& dst, const ModelPar& src) {
    static_assert(sizeof(ModelPar) % 4 == 0, "copied by words");
    for (int w = threadIdx.y * blockDim.x + threadIdx.x; w < (int)(sizeof(ModelPar) / 4); w += blockDim.x * blockDim.y)
        reinterpret_cast<int*>(&dst)[w] = reinterpret_cast<const int*>(&src)[w];
    __syncthreads();
}

struct ModelMaps {  // TMA descriptors of one model's interior sweeps (global memory, 64-byte aligned)
    VelMaps v;
    StrMaps s;
};

// dynamic shared memory of the kernels with interior tiles (1-D media only)
constexpr int VEL_RING = TMA_NS * VelSlot::ELEMS * (int)sizeof(float) + TMA_SMEM_PAD, STR_RING = str_ring_bytes<float, true>();

__device__ __forceinline__ bool item_live(const Work& it, const int* limit, const int* run_step, int ofs, int& m) {
    m = it.tm >> 8;
    return *run_step + ofs < limit[m];
}

template <bool STRESS, bool ANY>
__global__ void __launch_bounds__(PML_TILE, 4) k_bpml(const ModelDev* __restrict__ models,
                                                      const Work* __restrict__ work, int b0,
                                                      const int* __restrict__ limit, const int* run_step, int ofs,
                                                      int* gstatus) {
    __shared__ __align__(128) float sm[PML_TILE * (STRESS ? AUX_NS : AUX_NV)];
    __shared__ __align__(8) uint64_t bar;
    pdl_wait();
    pdl_launch_dependents();
    const Work it = work[b0 + blockIdx.x];
    int m;
    if (!item_live(it, limit, run_step, ofs, m)) return;
    __shared__ ModelPar M;
    load_par(M, models[m]);
    if (STRESS) str_pml_tile<float, false, ANY>(M.g, M.f, M.D, M.X, M.c, it.bx, sm, smem_addr(&bar), gstatus);
    else vel_pml_tile<float, false, ANY>(M.g, M.f, M.D, M.X, M.c, it.bx, sm, smem_addr(&bar), gstatus);
}

// A half-step of a small batch in one launch: the interior, fault-band and PML items (contiguous
// in the list by type), as k_vel_small / k_str_small do for one model.
template <bool STRESS, bool ANY>
__global__ void __launch_bounds__(256, 4) k_bhalf(const ModelDev* __restrict__ models, const ModelMaps* __restrict__ maps,
                                                  const Work* __restrict__ work, int b0, const int* __restrict__ limit,
                                                  const int* run_step, int ofs, int kchunk, int* gstatus) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* ring = reinterpret_cast<float*>(smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u));
    __shared__ __align__(8) uint64_t bars[TMA_NS];
    __shared__ ModelPar P;
    const Work it = work[b0 + blockIdx.x];
    pdl_wait();
    pdl_launch_dependents();
    int m;
    if (!item_live(it, limit, run_step, ofs, m)) return;
    const ModelDev& M = models[m];
    load_par(P, M);
    switch (it.tm & 255) {
        case W_VEL_INT:
        case W_STR_INT: {
            tma_ring_init(bars);
            if (STRESS)
                str_interior_tma_body<float, true>(maps[m].s, P.g, P.f, P.c, kchunk, it.bx, it.by, it.bz, ring, bars, gstatus);
            else
                vel_interior_tma_body<float, true>(maps[m].v, P.g, P.f, P.c, kchunk, it.bx, it.by, it.bz, ring, bars, gstatus);
            break;
        }
        case W_VEL_FAULT:
        case W_STR_FAULT:
            if (STRESS) str_fault_body<float>(P.g, P.f, M.q, P.c, it.bx, it.by, it.bz);
            else vel_fault_body<float>(P.g, P.f, M.q, P.c, M.law, M.fs, M.it_dev, M.status, it.bx, it.by, it.bz);
            break;
        default:
            if (STRESS) str_pml_tile<float, false, ANY>(P.g, P.f, P.D, P.X, P.c, it.bx, ring, smem_addr(bars), gstatus);
            else vel_pml_tile<float, false, ANY>(P.g, P.f, P.D, P.X, P.c, it.bx, ring, smem_addr(bars), gstatus);
    }
}

using BatchPmlKernel = void (*)(const ModelDev*, const Work*, int, const int*, const int*, int, int*);
using BatchHalfKernel = void (*)(const ModelDev*, const ModelMaps*, const Work*, int, const int*, const int*, int, int, int*);
// the same with ANY, in fd3d_forms.cu (see pml_kernel_forms)
BatchPmlKernel batch_pml_forms(bool stress);
BatchHalfKernel batch_half_forms(bool stress);

}  // namespace fd3d
