// Stage kernel with one thread per face, for grids too small to fill the
// GPU and for 1-D.
//
// A block owns a small box of cells.  It stages the box and its halo in
// shared memory; then every face of every direction has a thread of its own,
// which reconstructs both of its sides and evaluates the flux; then every
// cell has a thread, which adds its net flux and applies the stage.  The
// directions run side by side on different warps and the stage passes three
// barriers, so its latency is one reconstruction and one flux, where the
// tiled kernel runs them direction after direction.  A face's two
// reconstructions share their smoothness terms, so doing both costs little
// more than one (FP64 WENO2: 110 against 104 FP64 operations per face).  The
// boxes are sized so that each direction's faces fill whole warps.  KH 128^2,
// FP64, 32 RK3 steps: 1.19 -> 0.72 ms, 0.78 with code of its own for y (32^3,
// 16 steps: 11.6 -> 1.00 ms).
//
// The arithmetic and its order are those of stage_kernel, so the results
// are its bits.
#pragma once

#include "stage_kernel.cuh"

namespace als {

// Cells per block.  Faces per direction: 1-D 128; 2-D 119 and 128; 3-D 108,
// 120 and 128.
template<int DIM> struct FaceBox;
template<> struct FaceBox<1> {
    static constexpr int X = 127, Y = 1, Z = 1, B = 4;
};
template<> struct FaceBox<2> {
    static constexpr int X = 16, Y = 7, Z = 1, B = 2;
};
template<> struct FaceBox<3> {
    static constexpr int X = 8, Y = 4, Z = 3, B = 1;
};

// Resident blocks per SM the register budget is sized for (FP32 2-D, 256^2,
// 16 RK3 steps: 3 blocks 0.51 ms, 4 0.39, 5 0.43).
template<class R, int DIM>
__host__ __device__ constexpr int face_blocks() {
    return sizeof(R) == 4 && DIM == 2 ? 4 : FaceBox<DIM>::B;
}

template<class R, int DIM, int RECON, int FLUX>
struct FaceLayout {
    typedef FaceBox<DIM> Box;
    static constexpr int NV = DIM + 2;
    static constexpr int G = stage_ghosts(RECON, FLUX);
    static constexpr int TX = Box::X, TY = Box::Y, TZ = Box::Z;
    static constexpr int BX = TX + 2 * G;
    static constexpr int BY = DIM > 1 ? TY + 2 * G : 1;
    static constexpr int BZ = DIM > 2 ? TZ + 2 * G : 1;
    static constexpr int BOX = BX * BY * BZ;
    static constexpr int CELLS = TX * TY * TZ;
    static constexpr int GROUP = 128;   // threads per direction
    static constexpr int THREADS = DIM * GROUP;
    static constexpr size_t SMEM = sizeof(R) * size_t(NV) * (BOX + DIM * GROUP);
    static_assert((TX + 1) * TY * TZ <= GROUP && (DIM < 2 || TX * (TY + 1) * TZ <= GROUP) &&
        (DIM < 3 || TX * TY * (TZ + 1) <= GROUP) && CELLS <= THREADS, "a thread per face and per cell");
};

// Stencil values of a cell with the variables in another order: variable v
// is var[v] planes away.
template<class R>
struct OrderedFetch {
    const R* src;
    const int* var;
    int vstride;
    int s;
    __device__ __forceinline__ R at(int v, int o) const { return src[var[v] * vstride + o * s]; }
    __device__ __forceinline__ R dyn(int v, int o) const { return at(v, o); }
};

// In 2-D the y direction runs the code of the x direction with the momenta
// exchanged (a sum of two squares does not depend on their order), which
// halves the code a block has to fetch; three momenta, the sums of the
// entropy-conservative flux and FP32's contracted products do depend on it.
template<class R>
__host__ __device__ constexpr bool exchanges_momenta(int dim, int flux) {
    return sizeof(R) == 8 && dim == 2 && flux != FLUX_TECNO1;
}

// The face of thread i (0 <= i < GROUP) of direction `dir`, by the code of
// direction D: its flux into flx[v * GROUP + i], its wave speed into wmax
// where it counts.
template<class R, int DIM, int RECON, int FLUX, int KIND, int D>
__device__ __forceinline__ void face_of(const GridDesc& gd, R gamma, const R* box, R* flx, int i,
    int dir, R& wmax, int x0, int y0, int z0) {
    typedef FaceLayout<R, DIM, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int G = Lay::G;
    const int d0 = dir == 0 ? 1 : 0, d1 = dir == 1 ? 1 : 0, d2 = dir == 2 ? 1 : 0;
    const int f0 = Lay::TX + d0, f1 = Lay::TY + d1;
    if (i >= f0 * f1 * (Lay::TZ + d2)) {
        return;
    }
    const int fx = i % f0;
    const int fy = DIM > 1 ? (i / f0) % f1 : 0;
    const int fz = DIM > 2 ? i / (f0 * f1) : 0;
    const int s = dir == 0 ? 1 : (dir == 1 ? Lay::BX : Lay::BX * Lay::BY);
    // the cell to the face's right; the one to its left is s before it
    const R* right = box + ((DIM > 2 ? fz + G : 0) * Lay::BY + (DIM > 1 ? fy + G : 0)) * Lay::BX + fx + G;
    int var[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        var[v] = exchanges_momenta<R>(DIM, FLUX) && dir == 1 && (v == 1 || v == 2) ? 3 - v : v;
    }
    const OrderedFetch<R> fl{right - s, var, Lay::BOX, s};
    const OrderedFetch<R> fr{right, var, Lay::BOX, s};
    R ul[NV], ur[NV], skip[NV], F[NV];
    bool okl, okr;
    reconstruct_d<R, NV, RECON, true>(fl, skip, ul, gamma, okl);
    reconstruct_d<R, NV, RECON, true>(fr, ur, skip, gamma, okr);
    if (!okl || !okr) {
        reconstruct_f<R, NV, RECON>(fl, skip, ul, gamma);
        reconstruct_f<R, NV, RECON>(fr, ur, skip, gamma);
    }
    const R w = face_flux_best<R, DIM, FLUX, D>(ul, ur, gamma, F);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        flx[var[v] * Lay::GROUP + i] = F[v];
    }
    // the face counts when the cell to its left (or, first face, its own) and
    // its place across lie in the update region
    const bool valid = x0 + fx - d0 < gd.hi[0] && (DIM < 2 || y0 + fy - d1 < gd.hi[1]) &&
        (DIM < 3 || z0 + fz - d2 < gd.hi[2]);
    if (KIND == KIND_FLUX0 && valid && wmax < w) {
        wmax = w;
    }
}

template<class R, int DIM, int RECON, int FLUX, int KIND>
__device__ __forceinline__ void faces_tile(const StageParams& P, const LevelDesc& L, int tile,
    int member, unsigned char* smem) {
    typedef FaceLayout<R, DIM, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int G = Lay::G;
    constexpr int kind = KIND;
    constexpr bool last = kind == KIND_RK3_2 || kind == KIND_RK2_1;
    constexpr bool forms = kind == KIND_RK3_1 || kind == KIND_RK2_1;   // U1 formed on load
    const int tid = threadIdx.x;
    const GridDesc& gd = L.grid;
    StepState* st = L.state ? L.state + (L.subdomains ? 0 : member) : nullptr;

    R* box = reinterpret_cast<R*>(smem);
    R* flx = box + NV * Lay::BOX;

    const int tx = tile % gd.tiles[0];
    const int ty = (tile / gd.tiles[0]) % gd.tiles[1];
    const int tz = tile / (gd.tiles[0] * gd.tiles[1]);
    const int x0 = gd.lo[0] + tx * Lay::TX;
    const int y0 = gd.lo[1] + ty * Lay::TY;
    const int z0 = gd.lo[2] + tz * Lay::TZ;
    const long long base = (long long)member * L.member_stride;
    const R gamma = R(P.gamma);

    R c = R(0);
    if (forms) {
        if (st) {
            const double dt = step_dt(st);
            if (tile == 0 && tid == 0 && (member == 0 || !L.subdomains)) {
                st->dt = dt;
            }
            c = R(dt / st->dx[0]);
        } else {
            c = R(P.c_fixed);
        }
    } else if (kind == KIND_RK3_2) {
        c = st ? R(st->dt / st->dx[0]) : R(P.c_fixed);
    }

    const int sh = gd.ghosts - G;
    for (int b = tid; b < Lay::BOX; b += Lay::THREADS) {
        const int bx = b % Lay::BX;
        const int by = (b / Lay::BX) % Lay::BY;
        const int bz = b / (Lay::BX * Lay::BY);
        const int px = min(x0 + bx + sh, gd.N[0] - 1);
        const int py = DIM > 1 ? min(y0 + by + sh, gd.N[1] - 1) : 0;
        const int pz = DIM > 2 ? min(z0 + bz + sh, gd.N[2] - 1) : 0;
        const long long idx = base + ((long long)pz * gd.N[1] + py) * gd.N[0] + px;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            R val = static_cast<const R*>(L.in[v])[idx];
            if (forms) {
                val = val * c;
                val = val + static_cast<const R*>(L.un[v])[idx];
            }
            box[v * Lay::BOX + b] = val;
        }
    }
    __syncthreads();

    // the cell of this thread, and its U^n on its way early
    const int cx = tid % Lay::TX;
    const int cy = (tid / Lay::TX) % Lay::TY;
    const int cz = tid / (Lay::TX * Lay::TY);
    const int gx = x0 + cx, gy = y0 + cy, gz = z0 + cz;
    const bool cell = tid < Lay::CELLS && gx < gd.hi[0] && (DIM < 2 || gy < gd.hi[1]) &&
        (DIM < 3 || gz < gd.hi[2]);
    R un[NV];
    if (cell) {
        load_un<R, DIM, NV, KIND>(L, base, gx, gy, gz, un);
    }

    R wmax = R(0);
    const int group = tid / Lay::GROUP;
    const int face = tid % Lay::GROUP;
    R* mine = flx + group * NV * Lay::GROUP;
    if (exchanges_momenta<R>(DIM, FLUX) || group == 0) {
        face_of<R, DIM, RECON, FLUX, KIND, 0>(gd, gamma, box, mine, face, group, wmax, x0, y0, z0);
    } else if (DIM > 1 && group == 1) {
        face_of<R, DIM, RECON, FLUX, KIND, (DIM > 1 ? 1 : 0)>(gd, gamma, box, mine, face, 1, wmax, x0, y0, z0);
    } else if (DIM > 2) {
        face_of<R, DIM, RECON, FLUX, KIND, (DIM > 2 ? 2 : 0)>(gd, gamma, box, mine, face, 2, wmax, x0, y0, z0);
    }
    if (kind == KIND_FLUX0) {
        // a warp's faces share a direction
        const R w = warp_max(wmax);
        if ((tid & 31) == 0 && w > R(0)) {
            unsigned long long* dst = st ? &st->ws[group] : (L.ws_out + 3 * member + group);
            atomicMax(dst, (unsigned long long)__double_as_longlong(double(w)));
        }
    }
    __syncthreads();

    bool bad = false;
    long long bad_idx = 0;
    if (cell) {
        const int bidx = ((DIM > 2 ? cz + G : 0) * Lay::BY + (DIM > 1 ? cy + G : 0)) * Lay::BX + cx + G;
        R acc[NV], ub[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            ub[v] = box[v * Lay::BOX + bidx];
            acc[v] = R(0);
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const int f0 = Lay::TX + (d == 0 ? 1 : 0);
            const int f1 = Lay::TY + (d == 1 ? 1 : 0);
            const int l = (cz * f1 + cy) * f0 + cx;
            const int r = l + (d == 0 ? 1 : (d == 1 ? f0 : f0 * f1));
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const R tr = -flx[(d * NV + v) * Lay::GROUP + r];
                const R tl = -flx[(d * NV + v) * Lay::GROUP + l];
                acc[v] = acc[v] + (tr + (-tl));
            }
        }
        update_cell<R, DIM, NV, KIND>(P, L, member, base, c, gamma, acc, ub, un, gx, gy, gz, bad,
            bad_idx);
    }

    if (last && st) {
        if (bad) {
            atomicOr(&st->status, 1);
            atomicMin((unsigned long long*)&st->bad_index, (unsigned long long)bad_idx);
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            const unsigned int prev = atomicAdd(&st->arrive, 1u);
            const unsigned int tiles = unsigned(L.tiles_per_member) *
                (L.subdomains ? unsigned(L.members) : 1u);
            if (prev == tiles - 1) {
                __threadfence();
                finish_step(st);
            }
        }
    }
}

template<class R, int DIM, int RECON, int FLUX, int KIND>
__global__ void __launch_bounds__((FaceLayout<R, DIM, RECON, FLUX>::THREADS), (face_blocks<R, DIM>()))
faces_kernel(const StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    walk_work(P, [&](const LevelDesc& L, int tile, int member) {
        faces_tile<R, DIM, RECON, FLUX, KIND>(P, L, tile, member, smem);
    });
}

} // namespace als
