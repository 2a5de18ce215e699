// Host-side launch of the stage kernel for a run-time (reconstruction, flux,
// kind) triple.  Each translation unit that includes this header
// instantiates the kernels of one (precision, dimension) pair, so the heavy
// instantiations compile in parallel.
#pragma once

#include <algorithm>
#include <atomic>

#include <cuda_runtime.h>

#include "stage_faces.cuh"
#include "stage_kernel.cuh"
#include "stage_line.cuh"
#include "stage_rows.cuh"
#include "stage_zmarch.cuh"

namespace als {

// Blocks of KERNEL that the current device can hold at once.  A property of
// the kernel and the device: looked up once per device.
template<void (*KERNEL)(StageParams)>
cudaError_t resident_blocks(int threads, size_t smem, int* blocks) {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];
    int device = 0, sms = 0, per_sm = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) {
        return err;
    }
    const bool kept = device >= 0 && device < kDevices;
    if (kept && known[device].load(std::memory_order_relaxed) > 0) {
        *blocks = known[device].load(std::memory_order_relaxed);
        return cudaSuccess;
    }
    err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (err == cudaSuccess) {
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERNEL, threads, smem);
    }
    if (err != cudaSuccess) {
        return err;
    }
    *blocks = (per_sm < 1 ? 1 : per_sm) * sms;
    if (kept) {
        known[device].store(*blocks, std::memory_order_relaxed);
    }
    return cudaSuccess;
}

// One block per work item when the launch has no work counter; otherwise a
// persistent launch of as many blocks as can be resident at once (or
// `blocks_per_sm` per SM when > 0, capped by what fits), never more than
// there are work items.
//
// The solver's stages may be chained: a stage's blocks take their places while
// the one before it ends, which hides its launch (2 to 7 %).  With too few blocks for
// the GPU that costs more than it gives: the early ones double up on the SMs that the
// running stage leaves free, and the stage takes as long as those.  So a launch is chained
// from `quarters` quarters of the blocks that the GPU holds at once.  us per RK3 step,
// apart / chained: TeCNO6 256^2, 128 tiles, 119 / 190; FP64 faces 32^2 17.9 / 20.2, 160^2
// (230 boxes of 296) 23 / 22; 24^3 29 / 33 (144 of 148); FP32 16 x 16 tiles 320^2 (400 of
// 592) 27 / 30, 64 x 648 x 3 (492) 36 / 33.  Always chained: FP64 16 x 16 tiles (320^2 43 /
// 41) and the FP32 1-D and 2-D faces, which are bound by latency, so that sharing an SM
// costs them nothing (64^2: 18.2 / 17.5).  These are replayed graphs; in steps launched one by
// one (P.chained 2) the launch itself counts more, and all faces are chained (FP64, 4 steps:
// 26 x 28 x 2 126 / 110 us, 61 x 339 106 / 93).
template<void (*KERNEL)(StageParams)>
cudaError_t launch_stage_blocks(int threads, size_t smem, const StageParams& P, int blocks_per_sm,
    cudaStream_t stream, int quarters, bool faces = false) {
    if (faces && P.chained == 2) {
        quarters = 0;
    }
    // raising the dynamic shared-memory limit is idempotent and cheap; it is
    // done on every launch so that every device the process uses is covered
    cudaError_t err = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize,
        int(smem));
    if (err != cudaSuccess) {
        return err;
    }
    if (P.total_work <= 0) {
        return cudaSuccess;
    }
    int resident = 0;
    if (P.counter || (P.chained && quarters > 0)) {
        err = resident_blocks<KERNEL>(threads, smem, &resident);
        if (err != cudaSuccess) {
            return err;
        }
    }
    long long blocks = P.total_work;
    if (P.counter) {
        int device = 0, sms = 0;
        err = cudaGetDevice(&device);
        if (err == cudaSuccess) {
            err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        }
        if (err != cudaSuccess) {
            return err;
        }
        const long long wanted = blocks_per_sm > 0 ? (long long)blocks_per_sm * sms : resident;
        blocks = std::min(blocks, std::min<long long>(resident, wanted));
    }
    cudaLaunchAttribute chained;
    chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chained.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(unsigned(blocks));
    config.blockDim = dim3(unsigned(threads));
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &chained;
    config.numAttrs = P.chained && 4 * blocks >= (long long)quarters * resident ? 1 : 0;
    return cudaLaunchKernelEx(&config, KERNEL, P);
}

// The kernel of one (kernel id, kind): a thread per face for id kFacesKernel
// and for 1-D two-point fluxes; in 2-D id 0 with a two-point flux the warps
// marching along y; id kPlanesKernel the columns marching along z; else the tiled
// stage_kernel of that shape.
template<class R, int DIM, int RECON, int FLUX, int KIND, int SHAPE>
cudaError_t launch_stage_one(const StageParams& P, int b, cudaStream_t s) {
    if constexpr (SHAPE == kFacesKernel) {
        typedef FaceLayout<R, DIM, RECON, FLUX> Lay;
        return launch_stage_blocks<faces_kernel<R, DIM, RECON, FLUX, KIND>>(Lay::THREADS, Lay::SMEM,
            P, b, s, DIM == 3 ? 4 : (sizeof(R) == 4 ? 0 : 3), true);
    } else if constexpr (SHAPE == kPlanesKernel) {
        typedef ZLayout<R, RECON, FLUX> Lay;
        return launch_stage_blocks<zmarch_kernel<R, RECON, FLUX, KIND>>(Lay::THREADS, Lay::SMEM, P,
            b, s, 3);
    } else if constexpr (marches_rows(DIM, FLUX, SHAPE)) {
        typedef RowLayout<R, RECON, FLUX> Lay;
        // a block of the schedule stands for eight of these warps
        return launch_stage_blocks<rows_kernel<R, RECON, FLUX, KIND>>(32, Lay::SMEM, P, 8 * b, s, 3);
    } else {
        typedef StageLayout<R, DIM, RECON, FLUX, SHAPE> Lay;
        return launch_stage_blocks<stage_kernel<R, DIM, RECON, FLUX, KIND, SHAPE>>(Lay::THREADS,
            Lay::SMEM, P, b, s, DIM == 3 ? 4 : (DIM == 2 && SHAPE == 1 && sizeof(R) == 8 ? 0 : 3));
    }
}

template<class R, int DIM, int RECON, int FLUX, int SHAPE>
cudaError_t launch_stage_kind(int kind, const StageParams& P, int b, cudaStream_t s) {
    switch (kind) {
    case KIND_FLUX0: return launch_stage_one<R, DIM, RECON, FLUX, KIND_FLUX0, SHAPE>(P, b, s);
    case KIND_RK2_1: return launch_stage_one<R, DIM, RECON, FLUX, KIND_RK2_1, SHAPE>(P, b, s);
    case KIND_RK3_1: return launch_stage_one<R, DIM, RECON, FLUX, KIND_RK3_1, SHAPE>(P, b, s);
    case KIND_RK3_2: return launch_stage_one<R, DIM, RECON, FLUX, KIND_RK3_2, SHAPE>(P, b, s);
    default: return cudaErrorInvalidValue;
    }
}

// The kernel is a run-time choice among those built for the combination
// (kernel_built).
template<class R, int DIM, int RECON, int FLUX>
cudaError_t launch_stage_shape(int kernel, int kind, const StageParams& P, int b, cudaStream_t s) {
    if constexpr (kernel_built(DIM, RECON, FLUX, kFacesKernel)) {
        if (kernel == kFacesKernel) {
            return launch_stage_kind<R, DIM, RECON, FLUX, kFacesKernel>(kind, P, b, s);
        }
    }
    if constexpr (kernel_built(DIM, RECON, FLUX, kPlanesKernel)) {
        if (kernel == kPlanesKernel) {
            return launch_stage_kind<R, DIM, RECON, FLUX, kPlanesKernel>(kind, P, b, s);
        }
    }
    if constexpr (kernel_built(DIM, RECON, FLUX, 0)) {
        if (kernel == 0) {
            return launch_stage_kind<R, DIM, RECON, FLUX, 0>(kind, P, b, s);
        }
    }
    if constexpr (kernel_built(DIM, RECON, FLUX, 1)) {
        if (kernel == 1) {
            return launch_stage_kind<R, DIM, RECON, FLUX, 1>(kind, P, b, s);
        }
    }
    return cudaErrorInvalidValue;
}

template<class R, int DIM, int RECON>
cudaError_t launch_stage_flux(int flux, int kind, int shape, const StageParams& P, int b,
    cudaStream_t s) {
    switch (flux) {
    case FLUX_HLL: return launch_stage_shape<R, DIM, RECON, FLUX_HLL>(shape, kind, P, b, s);
    case FLUX_HLL3: return launch_stage_shape<R, DIM, RECON, FLUX_HLL3>(shape, kind, P, b, s);
    case FLUX_CENTRAL: return launch_stage_shape<R, DIM, RECON, FLUX_CENTRAL>(shape, kind, P, b, s);
    default: break;
    }
    // the TeCNO fluxes are built for reconstruction "none" only
    if constexpr (RECON == RECON_NONE) {
        switch (flux) {
        case FLUX_TECNO1: return launch_stage_shape<R, DIM, RECON, FLUX_TECNO1>(shape, kind, P, b, s);
        case FLUX_TECNO4: return launch_stage_shape<R, DIM, RECON, FLUX_TECNO4>(shape, kind, P, b, s);
        case FLUX_TECNO6: return launch_stage_shape<R, DIM, RECON, FLUX_TECNO6>(shape, kind, P, b, s);
        default: break;
        }
    }
    return cudaErrorInvalidValue;
}

// The reconstructions of a translation unit: the 2-D and 3-D kernels of one
// precision are built in three units, side by side (one alone takes minutes).
constexpr int kReconGroups = 3;
constexpr int recon_group(int recon) {
    return recon == RECON_NONE || recon == RECON_WENO2 || recon == RECON_ENO2 ? 0
        : (recon == RECON_ENO3 || recon == RECON_ENO4 || recon == RECON_WENO3 ? 1 : 2);
}

template<class R, int DIM, int GROUP>
cudaError_t launch_stage_group(int recon, int flux, int kind, int shape, const StageParams& P, int b,
    cudaStream_t s) {
    if constexpr (GROUP == 0) {
        switch (recon) {
        case RECON_NONE: return launch_stage_flux<R, DIM, RECON_NONE>(flux, kind, shape, P, b, s);
        case RECON_WENO2: return launch_stage_flux<R, DIM, RECON_WENO2>(flux, kind, shape, P, b, s);
        case RECON_ENO2: return launch_stage_flux<R, DIM, RECON_ENO2>(flux, kind, shape, P, b, s);
        default: return cudaErrorInvalidValue;
        }
    } else if constexpr (GROUP == 1) {
        switch (recon) {
        case RECON_ENO3: return launch_stage_flux<R, DIM, RECON_ENO3>(flux, kind, shape, P, b, s);
        case RECON_ENO4: return launch_stage_flux<R, DIM, RECON_ENO4>(flux, kind, shape, P, b, s);
        case RECON_WENO3: return launch_stage_flux<R, DIM, RECON_WENO3>(flux, kind, shape, P, b, s);
        default: return cudaErrorInvalidValue;
        }
    } else {
        switch (recon) {
        case RECON_MC: return launch_stage_flux<R, DIM, RECON_MC>(flux, kind, shape, P, b, s);
        case RECON_MM: return launch_stage_flux<R, DIM, RECON_MM>(flux, kind, shape, P, b, s);
        case RECON_WENOF2: return launch_stage_flux<R, DIM, RECON_WENOF2>(flux, kind, shape, P, b, s);
        default: return cudaErrorInvalidValue;
        }
    }
}

// A unit's entry point.
#define ALS_STAGE_ARGS int recon, int flux, int kind, int shape, const StageParams& P, int blocks_per_sm, cudaStream_t s
typedef cudaError_t (*StageLauncher)(ALS_STAGE_ARGS);

// The unit that holds the kernels of `recon`.
inline cudaError_t launch_stage_unit(const StageLauncher (&units)[kReconGroups], ALS_STAGE_ARGS) {
    return units[recon_group(recon)](recon, flux, kind, shape, P, blocks_per_sm, s);
}

// Whole steps of `members` 1-D lines, one cluster of `blocks` blocks each; with
// `clusters` only the number of clusters that can be resident at once.
#define ALS_LINE_ARGS bool rk3, const LineParams& P, int members, int blocks, cudaStream_t s, int* clusters
template<class R, int RECON, int FLUX, bool RK3>
cudaError_t launch_line_one(const LineParams& P, int members, int blocks, cudaStream_t stream,
    int* clusters) {
    const size_t smem = LineLayout<R, RECON, FLUX>::smem(P.stride);
    // a thread per face of the largest piece, up to the block's limit: the wide
    // block where it takes fewer passes (each a third longer), or shares SMs
    const int faces = P.stride - 2 * P.ghosts + 1;
    auto passes = [&](int threads) { return (faces + threads - 1) / threads; };
    const bool wide = faces > kLineThreads
        ? 13 * passes(kLineThreadsWide) < 10 * passes(kLineThreads)
        : (long long)members * blocks > 148;
    const int most = wide ? kLineThreadsWide : kLineThreads;
    const int threads = std::min((faces + 31) / 32 * 32, most);
    auto kernel = wide ? line_kernel<R, RECON, FLUX, RK3, kLineThreadsWide>
                       : line_kernel<R, RECON, FLUX, RK3, kLineThreads>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
        int(smem));
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = unsigned(blocks);
    cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(unsigned(members) * unsigned(blocks));
    config.blockDim = dim3(unsigned(threads));
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &cluster;
    config.numAttrs = 1;
    return clusters ? cudaOccupancyMaxActiveClusters(clusters, kernel, &config)
                    : cudaLaunchKernelEx(&config, kernel, P);
}

template<class R, int RECON, int FLUX>
cudaError_t launch_line_steps(ALS_LINE_ARGS) {
    return rk3 ? launch_line_one<R, RECON, FLUX, true>(P, members, blocks, s, clusters)
               : launch_line_one<R, RECON, FLUX, false>(P, members, blocks, s, clusters);
}

template<class R, int RECON>
cudaError_t launch_line_flux(int flux, ALS_LINE_ARGS) {
    switch (flux) {
    case FLUX_HLL: return launch_line_steps<R, RECON, FLUX_HLL>(rk3, P, members, blocks, s, clusters);
    case FLUX_HLL3: return launch_line_steps<R, RECON, FLUX_HLL3>(rk3, P, members, blocks, s, clusters);
    case FLUX_CENTRAL: return launch_line_steps<R, RECON, FLUX_CENTRAL>(rk3, P, members, blocks, s, clusters);
    default: return cudaErrorInvalidValue;
    }
}

template<class R>
cudaError_t launch_line(int recon, int flux, ALS_LINE_ARGS) {
    switch (recon) {
    case RECON_NONE: return launch_line_flux<R, RECON_NONE>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_WENO2: return launch_line_flux<R, RECON_WENO2>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_ENO2: return launch_line_flux<R, RECON_ENO2>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_ENO3: return launch_line_flux<R, RECON_ENO3>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_ENO4: return launch_line_flux<R, RECON_ENO4>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_MC: return launch_line_flux<R, RECON_MC>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_MM: return launch_line_flux<R, RECON_MM>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_WENOF2: return launch_line_flux<R, RECON_WENOF2>(flux, rk3, P, members, blocks, s, clusters);
    case RECON_WENO3: return launch_line_flux<R, RECON_WENO3>(flux, rk3, P, members, blocks, s, clusters);
    default: return cudaErrorInvalidValue;
    }
}

// Cells per work item of kernel `shape` (0 0 0 when it is not built for the
// dimension; the runs of the marching rows are split further by the host).
template<int DIM>
void stage_tile_dim(int shape, int* tile) {
    tile[0] = tile[1] = tile[2] = 0;
    if (shape == kFacesKernel) {
        tile[0] = FaceBox<DIM>::X;
        tile[1] = FaceBox<DIM>::Y;
        tile[2] = FaceBox<DIM>::Z;
    }
    if (shape == kPlanesKernel && DIM == 3) {
        tile[0] = kColumnsX;
        tile[1] = kColumnsY;
        tile[2] = ALS_ZMARCH_SEG;
    }
    if (shape == 0) {
        tile[0] = TileShape<DIM, 0>::X;
        tile[1] = TileShape<DIM, 0>::Y;
        tile[2] = TileShape<DIM, 0>::Z;
    }
    if constexpr (DIM >= 2) {
        if (shape == 1) {
            tile[0] = TileShape<DIM, 1>::X;
            tile[1] = TileShape<DIM, 1>::Y;
            tile[2] = TileShape<DIM, 1>::Z;
        }
    }
}

// Entry points defined by the per-(precision, dimension) translation units.
// `shape` selects the tile shape (shape_built), `blocks_per_sm` (0 = as
// many as fit) sizes the persistent grid.  stage_tile_* report the tile of
// a shape as the kernels of that unit were built, so the host always covers
// the grid with the tiles the kernels expect.
cudaError_t launch_stage_f64_1d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_2d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_2d_eno(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_2d_limiter(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_3d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_3d_eno(ALS_STAGE_ARGS);
cudaError_t launch_stage_f64_3d_limiter(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_1d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_2d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_2d_eno(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_2d_limiter(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_3d(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_3d_eno(ALS_STAGE_ARGS);
cudaError_t launch_stage_f32_3d_limiter(ALS_STAGE_ARGS);
cudaError_t launch_line_f64(int recon, int flux, ALS_LINE_ARGS);
cudaError_t launch_line_f32(int recon, int flux, ALS_LINE_ARGS);
void stage_tile_f64_1d(int shape, int* tile);
void stage_tile_f64_2d(int shape, int* tile);
void stage_tile_f64_3d(int shape, int* tile);
void stage_tile_f32_1d(int shape, int* tile);
void stage_tile_f32_2d(int shape, int* tile);
void stage_tile_f32_3d(int shape, int* tile);

} // namespace als
