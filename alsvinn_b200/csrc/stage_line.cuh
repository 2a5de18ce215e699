// Whole time steps of 1-D grids in one launch.
//
// A 1-D grid is too small for a launch per stage: 1024 cells are a few
// blocks, and a stage takes its latency whatever the GPU's width.  Here a
// thread-block cluster owns one member for as many steps as the host asks
// for.  Each of its blocks keeps a piece of the line in shared memory (U^n,
// the unscaled flux L, and the inputs of the later stages, each with its
// ghost cells); an updated cell is written straight into the ghost cells of
// the neighbouring block through distributed shared memory, and stages are
// separated by cluster barriers instead of launches: three per RK3 step, the
// first of which also carries the step's wave-speed maximum to every block.
// What a block tells the others (speeds, a bad cell) it stores into a slot of
// its own in each of them: all accesses to another block's shared memory are plain
// stores through mapped pointers.  They are in bounds because a piece holds its own
// cells and G ghost cells a side (a cell within G of a piece's end goes to one place
// of one neighbour, or to the first or last piece's ghosts), and in time because the
// cluster waits before the first of them and after the last, and leaves early, on the
// member's `done`, only as a whole.  Sod, 1024 cells, HLL, RK3 to T = 0.2 (498
// steps): 3.44 ms, 2.3 us a stage; with a launch per stage 7.97 ms.
//
// The arithmetic and its order are those of the other stage kernels
// (face_of, update_cell, finish_step), so the results are their bits.
#pragma once

#include <cooperative_groups.h>

#include "stage_kernel.cuh"

namespace als {

// The member's line and clock for one launch.
struct LineParams {
    const void* in;          // U^n of member 0, variable planes one after another
    void* even;              // where a member that takes an even number of steps leaves its state
    void* odd;               // and after an odd number (RK2 alternates buffers)
    StepState* state;
    long long plane;         // padded cells per plane
    int n;                   // interior cells
    int ghosts;              // ghost cells per side
    int bc;
    int steps;               // most steps of this launch
    int stride;              // padded cells of a block's piece, at most
    double gamma;
};

// Most threads of a block.  The kernel is built for two numbers: 256 threads may
// have 255 registers each (FP64 uses 194), 288, the 257 faces of 256 cells in one
// pass, share a quarter of the SM's registers three warps at a time (168 each,
// which also lets more blocks share an SM).  FP64 WENO2, us per RK3 step, 256 / 288: 1
// line of 1024 cells in pieces of 128 7.3 / 7.4, of 256 9.2 / 8.4, 148 lines in pieces
// of 512 12.5 / 11.7, of 1024 18.5 / 19.8; 4096 lines of 128 cells 190 / 108.
constexpr int kLineThreads = 256;
constexpr int kLineThreadsWide = 288;
constexpr int kLineBlocks = 8;        // blocks per cluster, at most (the portable size)
constexpr int kLineCells = 1024;      // cells of a block's piece, at most

template<class R, int RECON, int FLUX>
struct LineLayout {
    static constexpr int NV = 3;
    static constexpr int G = stage_ghosts(RECON, FLUX);
    // U^n, L, stage inputs 1 and 2, fluxes
    static size_t smem(int stride) {
        return sizeof(R) * size_t(NV) * (4 * size_t(stride) + size_t(stride + 1));
    }
};

// Largest of 32 lanes' non-negative doubles, as bits (their order is that of
// the integers): the high words first, then the low words of those that tie.
__device__ __forceinline__ unsigned long long warp_max_bits(double w) {
    const unsigned hi = unsigned(__double2hiint(w));
    const unsigned top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? unsigned(__double2loint(w)) : 0u);
    return ((unsigned long long)top << 32) | lo;
}

template<class R, int RECON, int FLUX, bool RK3, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) line_kernel(const LineParams P) {
    namespace cg = cooperative_groups;
    typedef LineLayout<R, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int G = Lay::G;
    extern __shared__ __align__(16) unsigned char smem[];
    // every block's wave-speed maximum and first bad cell of the step, written
    // by that block into all of them; this block's own before it is sent
    __shared__ unsigned long long speeds[kLineBlocks], bads[kLineBlocks];
    __shared__ unsigned long long my_speed[2], my_bad;

    cg::cluster_group cluster = cg::this_cluster();
    const int blocks = int(cluster.num_blocks());
    const int rank = int(cluster.block_rank());
    const int member = int(blockIdx.x) / blocks;
    const int tid = threadIdx.x;
    const int threads = blockDim.x;
    StepState* st = P.state + member;
    if (((const volatile StepState*)st)->done) {
        return;   // the whole cluster
    }
    const int begin = int((long long)P.n * rank / blocks);
    const int end = int((long long)P.n * (rank + 1) / blocks);
    const int m = end - begin;
    const int stride = P.stride;
    R* un = reinterpret_cast<R*>(smem);
    R* lf = un + NV * stride;       // L
    R* u1 = lf + NV * stride;
    R* u2 = u1 + NV * stride;
    R* flx = u2 + NV * stride;      // flux through the left face of cell i
    const R gamma = R(P.gamma);
    const long long base = (long long)member * NV * P.plane;

    if (tid == 0) {
        my_speed[0] = 0;
        my_speed[1] = 0;
        my_bad = ~0ull;
    }
    for (int i = tid; i < m + 2 * G; i += threads) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            un[v * stride + i] = (static_cast<const R*>(P.in) + base)[v * P.plane + begin + i +
                P.ghosts - G];
        }
    }
    double t = st->t;
    double dt = st->dt;
    long long steps = st->steps;
    const long long max_steps = st->max_steps;
    const double end_time = st->end_time;
    int status = st->status;
    long long bad_step = st->bad_step;
    unsigned long long bad_cell = ~0ull;
    cluster.sync();

    // flux through every face of the piece (face i: left of cell i)
    auto faces = [&](const R* u, double& wmax) {
        for (int i = tid; i <= m; i += threads) {
            const StridedFetch<R, int> fl{u + G + i - 1, stride, 1};
            const StridedFetch<R, int> fr{u + G + i, stride, 1};
            R ul[NV], ur[NV], skip[NV], F[NV];
            bool okl, okr;
            reconstruct_d<R, NV, RECON, true>(fl, skip, ul, gamma, okl);
            reconstruct_d<R, NV, RECON, true>(fr, ur, skip, gamma, okr);
            if (!okl || !okr) {
                reconstruct_f<R, NV, RECON>(fl, skip, ul, gamma);
                reconstruct_f<R, NV, RECON>(fr, ur, skip, gamma);
            }
            const R w = face_flux_best<R, 1, FLUX, 0>(ul, ur, gamma, F);
            if (wmax < double(w)) {
                wmax = double(w);
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                flx[v * (stride + 1) + i] = F[v];
            }
        }
    };
    auto net = [&](int i, R* acc) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const R tr = -flx[v * (stride + 1) + i + 1];
            const R tl = -flx[v * (stride + 1) + i];
            acc[v] = R(0) + (tr + (-tl));
        }
    };
    // cell i's value into array `to`: its own place, the ghost cells of the
    // neighbouring blocks, and its boundary images
    auto store = [&](R* to, int i, const R* val) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            to[v * stride + i + G] = val[v];
        }
        if (i >= G && i < m - G) {
            return;
        }
        auto send = [&](int r, int at) {
            R* far = cluster.map_shared_rank(to, r);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                far[v * stride + at] = val[v];
            }
        };
        if (i < G && rank > 0) {
            const int first = int((long long)P.n * (rank - 1) / blocks);
            send(rank - 1, begin - first + i + G);
        }
        if (i >= m - G && rank < blocks - 1) {
            send(rank + 1, i - m + G);
        }
        int pos[3] = {0, 0, 0};
        const int images = boundary_images(begin + i, P.n, G, P.bc, pos);
        for (int k = 1; k < images; ++k) {
            const int last = int((long long)P.n * (blocks - 1) / blocks);
            if (pos[k] < G) {
                send(0, pos[k]);
            } else {
                send(blocks - 1, pos[k] - last);
            }
        }
    };

    int taken = 0;
    for (; taken < P.steps;) {
        // L(U^n) and the wave speeds
        double wmax = 0;
        faces(un, wmax);
        const unsigned long long w = warp_max_bits(wmax);
        if ((tid & 31) == 0) {
            atomicMax(&my_speed[taken & 1], w);
        }
        __syncthreads();
        if (tid < blocks) {
            cluster.map_shared_rank(speeds, tid)[rank] = my_speed[taken & 1];
        }
        for (int i = tid; i < m; i += threads) {
            R acc[NV];
            net(i, acc);
            store(lf, i, acc);
        }
        cluster.sync();
        if (tid == 0) {
            my_speed[(taken & 1) ^ 1] = 0;   // the next step's
        }
        unsigned long long top = 0;
        for (int r = 0; r < blocks; ++r) {
            top = speeds[r] > top ? speeds[r] : top;
        }
        const double ws[3] = {__longlong_as_double((long long)top), 0.0, 0.0};
        dt = step_dt_of(ws, st->dx, st->cfl, end_time, t);
        const R c = R(dt / st->dx[0]);
        for (int i = tid; i < m + 2 * G; i += threads) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                R x = lf[v * stride + i] * c;
                u1[v * stride + i] = x + un[v * stride + i];
            }
        }
        __syncthreads();
        double unused = 0;
        if (RK3) {
            faces(u1, unused);
            __syncthreads();
            for (int i = tid; i < m; i += threads) {
                R val[NV];
                net(i, val);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    val[v] = combine_stage<R, KIND_RK3_1>(val[v], c, u1[v * stride + i + G],
                        un[v * stride + i + G]);
                }
                store(u2, i, val);
            }
            cluster.sync();
        }
        const R* last = RK3 ? u2 : u1;
        faces(last, unused);
        if (RK3) {
            __syncthreads();
        } else {
            // neighbours form u1 from the ghost cells of un that are written next
            cluster.sync();
        }
        for (int i = tid; i < m; i += threads) {
            R val[NV];
            net(i, val);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                val[v] = combine_stage<R, RK3 ? KIND_RK3_2 : KIND_RK2_1>(val[v], c,
                    last[v * stride + i + G], un[v * stride + i + G]);
            }
            store(un, i, val);
            if (!obeys_constraints<R, NV>(val, gamma)) {
                atomicMin(&my_bad, (unsigned long long)(begin + i + P.ghosts));
            }
        }
        __syncthreads();
        if (tid < blocks) {
            cluster.map_shared_rank(bads, tid)[rank] = my_bad;
        }
        cluster.sync();
        for (int r = 0; r < blocks; ++r) {
            bad_cell = bads[r] < bad_cell ? bads[r] : bad_cell;
        }
        t = t + dt;
        steps = steps + 1;
        ++taken;
        if (bad_cell != ~0ull) {
            status = 1;
            bad_step = bad_step < 0 ? steps : bad_step;
        }
        if (t >= end_time || status != 0 || steps >= max_steps) {
            break;
        }
    }

    R* out = static_cast<R*>((taken & 1) ? P.odd : P.even) + base;
    const int from = rank == 0 ? 0 : G;
    const int to = m + G + (rank == blocks - 1 ? G : 0);
    for (int i = from + tid; i < to; i += threads) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            out[v * P.plane + begin + i + P.ghosts - G] = un[v * stride + i];
        }
    }
    if (rank == 0 && tid == 0) {
        st->t = t;
        st->dt = dt;
        st->steps = steps;
        st->status = status;
        st->bad_step = bad_step;
        if (bad_cell != ~0ull) {
            st->bad_index = (long long)bad_cell;
        }
        st->done = t >= end_time || status != 0 || steps >= max_steps ? 1 : 0;
    }
    // no block leaves while another may still write into its shared memory
    cluster.sync();
}

} // namespace als
