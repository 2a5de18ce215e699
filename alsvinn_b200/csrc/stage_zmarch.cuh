// 3-D stage kernel that marches along z (tile shape 1 of the 3-D stage).
//
// A block owns a 16 x 15 column of cells over a segment of at most
// ALS_ZMARCH_SEG cells along z (the host chooses the length).  It keeps a ring
// of three x-y planes (each with its x-y halo of G cells, every conserved
// variable) in shared memory and walks the segment plane by plane.  Per plane
// every x face and then every y face has a thread, which reconstructs both of
// its sides and evaluates the flux; then the thread of each column
// reconstructs the next cell of its column along z and evaluates the z face
// between the two, keeping that face's flux and the next cell's right state
// (in shared memory, private to the column) for the next plane.  So every cell
// is reconstructed along z once and every z face is evaluated once, where the
// 8 x 8 x 4 tiles of shape 0 reconstruct 1.5 cells per cell along z and stage a
// box of 4.5 times the tile.  The columns are 16 x 15 so that 255 x faces, 256 y
// faces and 240 columns fill 256 threads, which leaves FP64 128 registers at
// two blocks per SM.  KH 128^3 x 2, FP64, 4 RK3 steps: 6.72 ms, with 16 x 16
// columns, 288 threads and each cell reconstructed once per direction through
// shared memory (six barriers a plane instead of three) 7.65.
//
// The arithmetic and its order are those of stage_kernel (the same
// reconstruction, flux and update_cell; the net flux of a cell adds its x,
// then y, then z contribution), so the two shapes give the same bits.  Built
// for reconstructions whose stencil reaches one cell each way along z
// (WENO2, ENO2, MC, MM, WENOF2, none) and the two-point fluxes.
#pragma once

#include "stage_kernel.cuh"

namespace als {

template<class R, int RECON, int FLUX>
struct ZLayout {
    static constexpr int NV = 5;
    static constexpr int G = stage_ghosts(RECON, FLUX);
    static constexpr int S = recon_ghosts(RECON) - 1;   // stencil half-width along z
    static constexpr int TX = kColumnsX;
    static constexpr int TY = kColumnsY;
    static constexpr int BX = TX + 2 * G;
    static constexpr int BY = TY + 2 * G;
    static constexpr int PLANE = BX * BY;
    static constexpr int RING = 3;
    static constexpr int COLS = TX * TY;
    static constexpr int THREADS = 256;
    static constexpr int FACX = (TX + 1) * TY;
    static constexpr int FACY = TX * (TY + 1);
    // ring, x and y face fluxes, and per column the right state below the next
    // z face and the flux through the face below
    static constexpr size_t SMEM = sizeof(R) *
        (size_t(NV) * PLANE * RING + size_t(NV) * (FACX + FACY) + size_t(2 * NV) * COLS);
    static constexpr int BLOCKS = ALS_ZMARCH_BLOCKS;
    static_assert(S == 0 || S == 1, "the ring holds a stencil of one cell each way along z");
    static_assert(COLS <= THREADS && FACX <= THREADS && FACY <= THREADS, "a thread per column and face");
    static_assert(BLOCKS * (SMEM + 1024) <= 228 * 1024, "the blocks share the SM's memory");
};

// Values of one column at planes kc-1, kc, kc+1 of the ring (the fetcher of
// reconstruct_f along z; offsets beyond one cell are never asked for).
template<class R>
struct ColumnFetch {
    const R* m;
    const R* c;
    const R* p;
    int vstride;
    __device__ __forceinline__ R at(int v, int o) const {
        return (o < 0 ? m : (o > 0 ? p : c))[v * vstride];
    }
    __device__ __forceinline__ R dyn(int v, int o) const { return at(v, o); }
};

// The x (D = 0) or y (D = 1) faces of plane `pl`, a thread each: both sides
// reconstructed (they share their smoothness terms) and the flux into
// flx[v * faces + i].
template<class R, int RECON, int FLUX, int KIND, int D>
__device__ __forceinline__ void plane_faces(const GridDesc& gd, R gamma, const R* pl, R* flx,
    R& wmax, int x0, int y0) {
    typedef ZLayout<R, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int F0 = Lay::TX + (D == 0 ? 1 : 0);
    constexpr int FC = D == 0 ? Lay::FACX : Lay::FACY;
    constexpr int ST = D == 0 ? 1 : Lay::BX;
    const int i = threadIdx.x;
    if (i >= FC) {
        return;
    }
    const int fx = i % F0;
    const int fy = i / F0;
    const R* right = pl + (fy + Lay::G) * Lay::BX + fx + Lay::G;
    const StridedFetch<R, int> fl{right - ST, Lay::PLANE, ST};
    const StridedFetch<R, int> fr{right, Lay::PLANE, ST};
    R ul[NV], ur[NV], skip[NV], F[NV];
    bool okl, okr;
    reconstruct_d<R, NV, RECON, true>(fl, skip, ul, gamma, okl);
    reconstruct_d<R, NV, RECON, true>(fr, ur, skip, gamma, okr);
    if (!okl || !okr) {
        reconstruct_f<R, NV, RECON>(fl, skip, ul, gamma);
        reconstruct_f<R, NV, RECON>(fr, ur, skip, gamma);
    }
    const R w = face_flux_best<R, 3, FLUX, D>(ul, ur, gamma, F);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        flx[v * FC + i] = F[v];
    }
    if (KIND == KIND_FLUX0) {
        const bool valid = x0 + fx - (D == 0 ? 1 : 0) < gd.hi[0] && y0 + fy - (D == 1 ? 1 : 0) < gd.hi[1];
        if (valid && wmax < w) {
            wmax = w;
        }
    }
}

// One work item: columns (tx, ty) over z segment tz of member `member`.
template<class R, int RECON, int FLUX, int KIND>
__device__ __forceinline__ void zmarch_tile(const StageParams& P, const LevelDesc& L, int tile,
    int member, unsigned char* smem) {
    typedef ZLayout<R, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int G = Lay::G;
    constexpr bool LAST = KIND == KIND_RK3_2 || KIND == KIND_RK2_1;
    const int tid = threadIdx.x;
    const GridDesc& gd = L.grid;
    StepState* st = L.state ? L.state + (L.subdomains ? 0 : member) : nullptr;

    R* ring = reinterpret_cast<R*>(smem);
    R* flx = ring + Lay::RING * NV * Lay::PLANE;
    R* fly = flx + NV * Lay::FACX;
    // column-private: Rk[v] = zs[v * COLS + col], Fm[v] = zs[(NV + v) * COLS + col]
    R* zs = fly + NV * Lay::FACY;

    const int tx = tile % gd.tiles[0];
    const int ty = (tile / gd.tiles[0]) % gd.tiles[1];
    const int tz = tile / (gd.tiles[0] * gd.tiles[1]);
    const int x0 = gd.lo[0] + tx * Lay::TX;
    const int y0 = gd.lo[1] + ty * Lay::TY;
    // segment tz of gd.tiles[2], which split the planes evenly
    const int nz = gd.hi[2] - gd.lo[2];
    const int k0 = gd.lo[2] + int((long long)nz * tz / gd.tiles[2]);
    const int k1 = gd.lo[2] + int((long long)nz * (tz + 1) / gd.tiles[2]);
    const long long base = (long long)member * L.member_stride;
    auto inp = [&](int v) { return static_cast<const R*>(L.in[v]) + base; };
    auto unp = [&](int v) { return static_cast<const R*>(L.un[v]) + base; };
    const R gamma = R(P.gamma);

    R c = R(0);
    if (KIND == KIND_RK2_1 || KIND == KIND_RK3_1) {
        if (st) {
            const double dt = step_dt(st);
            if (tile == 0 && tid == 0 && (member == 0 || !L.subdomains)) {
                st->dt = dt;
            }
            c = R(dt / st->dx[0]);
        } else {
            c = R(P.c_fixed);
        }
    } else if (KIND == KIND_RK3_2) {
        c = st ? R(st->dt / st->dx[0]) : R(P.c_fixed);
    }

    // plane k (interior index along z, -2 <= k <= n + 1) into its ring slot,
    // with the x-y halo; U1 = (dt/dx) L + U^n formed on load as in stage_tile
    const int sh = gd.ghosts - G;
    auto slot = [&](int k) { return ring + ((k - k0 + 3) % 3) * (NV * Lay::PLANE); };
    auto load_plane = [&](int k) {
        R* dst = slot(k);
        // cells beyond the planes read the nearest column, row or plane:
        // ordinary values, whose results nobody uses
        const int pz = max(0, min(k + gd.ghosts, gd.N[2] - 1));
        for (int b = tid; b < Lay::PLANE; b += Lay::THREADS) {
            const int bx = b % Lay::BX;
            const int by = b / Lay::BX;
            const int px = min(x0 + bx + sh, gd.N[0] - 1);
            const int py = min(y0 + by + sh, gd.N[1] - 1);
            const long long idx = ((long long)pz * gd.N[1] + py) * gd.N[0] + px;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                R val = inp(v)[idx];
                if (KIND == KIND_RK2_1 || KIND == KIND_RK3_1) {
                    val = val * c;
                    val = val + unp(v)[idx];
                }
                dst[v * Lay::PLANE + b] = val;
            }
        }
    };

    // this thread's column (threads past the columns help in the x-y phases)
    const bool column = tid < Lay::COLS;
    const int cx = tid % Lay::TX;
    const int cy = (tid / Lay::TX) % Lay::TY;
    const int coff = (cy + G) * Lay::BX + cx + G;
    const bool in_region = column && x0 + cx < gd.hi[0] && y0 + cy < gd.hi[1];
    // reconstruction of cell kc of this column along z
    auto recon_z = [&](int kc, R* l, R* r) {
        ColumnFetch<R> f{slot(kc - 1) + coff, slot(kc) + coff, slot(kc + 1) + coff, Lay::PLANE};
        reconstruct_f<R, NV, RECON>(f, l, r, gamma);
    };

    R wmax[3] = {R(0), R(0), R(0)};
    // the column's right state below the next z face, and the z flux below
    // the current cell, kept in shared memory between planes
    R* Rk = zs + (column ? tid : 0);
    R* Fm = zs + NV * Lay::COLS + (column ? tid : 0);
    {
        load_plane(k0 - 2);
        load_plane(k0 - 1);
        load_plane(k0);
        __syncthreads();
        if (column) {
            R l[NV], r[NV];
            recon_z(k0 - 1, l, r);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                Rk[v * Lay::COLS] = r[v];
            }
        }
        __syncthreads();
        load_plane(k0 + 1);
        __syncthreads();
        if (column) {
            R l[NV], r[NV], rb[NV], F[NV];
            recon_z(k0, l, r);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                rb[v] = Rk[v * Lay::COLS];
            }
            const R w = face_flux_best<R, 3, FLUX, 2>(rb, l, gamma, F);
            if (KIND == KIND_FLUX0 && in_region && wmax[2] < w) {
                wmax[2] = w;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                Fm[v * Lay::COLS] = F[v];
                Rk[v * Lay::COLS] = r[v];
            }
        }
    }

    bool bad = false;
    long long bad_idx = 0;
    for (int k = k0; k < k1; ++k) {
        __syncthreads();
        load_plane(k + 2);
        __syncthreads();
        const R* pl = slot(k);
        plane_faces<R, RECON, FLUX, KIND, 0>(gd, gamma, pl, flx, wmax[0], x0, y0);
        plane_faces<R, RECON, FLUX, KIND, 1>(gd, gamma, pl, fly, wmax[1], x0, y0);
        __syncthreads();
        if (column) {
            R acc[NV];
            const int xl = cy * (Lay::TX + 1) + cx;
            const int yl = cy * Lay::TX + cx;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const R xr = -flx[v * Lay::FACX + xl + 1];
                const R xf = -flx[v * Lay::FACX + xl];
                acc[v] = R(0) + (xr + (-xf));
                const R yr = -fly[v * Lay::FACY + yl + Lay::TX];
                const R yf = -fly[v * Lay::FACY + yl];
                acc[v] = acc[v] + (yr + (-yf));
            }
            // z: the face above the cell, between it and the next cell up
            R l[NV], r[NV], rb[NV], Fp[NV];
            recon_z(k + 1, l, r);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                rb[v] = Rk[v * Lay::COLS];
            }
            const R w = face_flux_best<R, 3, FLUX, 2>(rb, l, gamma, Fp);
            if (KIND == KIND_FLUX0 && in_region && wmax[2] < w) {
                wmax[2] = w;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const R tr = -Fp[v];
                const R tl = -Fm[v * Lay::COLS];
                acc[v] = acc[v] + (tr + (-tl));
                Fm[v * Lay::COLS] = Fp[v];
                Rk[v * Lay::COLS] = r[v];
            }
            if (in_region) {
                R ub[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    ub[v] = pl[v * Lay::PLANE + coff];
                }
                R un[NV];
                load_un<R, 3, NV, KIND>(L, base, x0 + cx, y0 + cy, k, un);
                update_cell<R, 3, NV, KIND>(P, L, member, base, c, gamma, acc, ub, un, x0 + cx, y0 + cy,
                    k, bad, bad_idx);
            }
        }
    }

    if (KIND == KIND_FLUX0) {
        __shared__ double wsh[3][Lay::THREADS / 32];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const R w = warp_max(wmax[d]);
            if ((tid & 31) == 0) {
                wsh[d][tid >> 5] = double(w);
            }
        }
        __syncthreads();
        if (tid < 3) {
            double m = 0;
            for (int q = 0; q < Lay::THREADS / 32; ++q) {
                m = fmax(m, wsh[tid][q]);
            }
            unsigned long long* dst = st ? &st->ws[tid] : (L.ws_out + 3 * member + tid);
            atomicMax(dst, (unsigned long long)__double_as_longlong(m));
        }
    }

    if (LAST && st) {
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

template<class R, int RECON, int FLUX, int KIND>
__global__ void __launch_bounds__((ZLayout<R, RECON, FLUX>::THREADS),
    (ZLayout<R, RECON, FLUX>::BLOCKS))
zmarch_kernel(const StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    walk_work(P, [&](const LevelDesc& L, int tile, int member) {
        zmarch_tile<R, RECON, FLUX, KIND>(P, L, tile, member, smem);
    });
}

} // namespace als
