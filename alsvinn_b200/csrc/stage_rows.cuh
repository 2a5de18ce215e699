// 2-D stage kernel whose warps march along y (tile shape 0 of the 2-D stage
// for the two-point fluxes).
//
// A block is one warp.  It owns 32 columns (one per lane) over a run of at
// most 32 rows and waits for nobody.  It keeps the rows the stencil needs in
// a ring in shared memory and walks the run row by row:
//   y  the lane reconstructs the next cell of its column from the ring and
//      evaluates the face between the two cells, keeping that face's flux
//      and the cell's right state in registers for the next row;
//   x  the lane reconstructs its cell of the current row, takes the left
//      state of the cell to its right from the next lane, evaluates the face
//      between them, and takes the flux of its left face from the lane
//      before.  What lies outside the 32 columns (the flux through the first
//      column's left face, the left state beyond the last column) is formed
//      for all rows of the run at once, one row per lane, before the walk.
// So the reconstructed states and fluxes stay in registers, there is no
// block barrier.  FP64 WENO2 + HLL3, per cell and stage: 670 to 701 FP64
// instructions of 1,207 to 1,292 (the tiled kernel with plain divisions: 895 of
// 2,650); FP64 pipe 55 to 58 % busy; FP32 620 to 710, 70 to 76 % of the issue
// slots.  Ms per RK3 step: KH
// 1024^2 FP64 0.279 (tiled) -> 0.235, 4096^2 4.66 (tiled, plain divisions) -> 2.83,
// 512 x 256^2 FP32 members 4.35 -> 2.21.
//
// Measured (KH 1024^2): 12 warps per SM with 166 registers 0.235, 16 with 128
// 0.235 (spills, and 1 to 2 % slower on larger grids), 18 with 96 0.260; x and y
// interleaved for more independent work per lane 0.248 to 0.258; forming U1
// as the rows are loaded instead of as they are stored 0.248.
//
// The arithmetic and its order are those of stage_kernel, so the results are
// its bits.
#pragma once

#include "stage_kernel.cuh"

namespace als {

template<class R, int RECON, int FLUX>
struct RowLayout {
    static constexpr int NV = 4;
    static constexpr int G = stage_ghosts(RECON, FLUX);
    static constexpr int S = recon_ghosts(RECON) - 1;   // stencil half-width
    static constexpr int TX = kRunColumns;
    static constexpr int RING = 2 * S + 1 > 2 ? 2 * S + 1 : 2;
    static constexpr int BX = TX + 2 * S;
    static constexpr int ROW = NV * BX;
    // ring; then per row of the run: right state left of the first column
    // (replaced by the flux through its left face), left state of the first
    // column, left state right of the last column
    static constexpr int HALO = NV * kRunRows;
    static constexpr size_t SMEM = sizeof(R) * size_t(RING * ROW + 3 * HALO);
    static_assert(TileShape<2, 0>::X == TX, "the tiles along x are the warps' columns");
};

#ifndef ALS_ROWS_WARPS64
#define ALS_ROWS_WARPS64 12
#endif
#ifndef ALS_ROWS_WARPS32
#define ALS_ROWS_WARPS32 24
#endif
// Resident warps per SM the register budget is sized for.
template<class R>
__host__ __device__ constexpr int rows_warps_per_sm() {
    return sizeof(R) == 8 ? ALS_ROWS_WARPS64 : ALS_ROWS_WARPS32;
}

// Values of a stage's input state straight from its planes, neighbours along
// x.
template<class R, int KIND>
struct StageInputFetch {
    const LevelDesc* L;
    long long cell;   // member offset + padded cell index
    R c;
    __device__ __forceinline__ R at(int v, int o) const {
        R val = static_cast<const R*>(L->in[v])[cell + o];
        if (KIND == KIND_RK2_1 || KIND == KIND_RK3_1) {
            val = val * c;
            val = val + static_cast<const R*>(L->un[v])[cell + o];
        }
        return val;
    }
    __device__ __forceinline__ R dyn(int v, int o) const { return at(v, o); }
};

// Stencil values of the lane's column from the ring (offset o along y).
template<class R, int RING, int ROW, int BX>
struct RingFetch {
    const R* ring;   // the lane's column in slot 0
    int slot;        // slot of the centre row
    __device__ __forceinline__ R at(int v, int o) const {
        int s = slot + o;
        s = s < 0 ? s + RING : (s >= RING ? s - RING : s);
        return ring[s * ROW + v * BX];
    }
    __device__ __forceinline__ R dyn(int v, int o) const { return at(v, o); }
};

// One work item: run `tile` of member `member`.
template<class R, int RECON, int FLUX, int KIND>
__device__ __forceinline__ void rows_tile(const StageParams& P, const LevelDesc& L, int tile,
    int member, unsigned char* smem) {
    typedef RowLayout<R, RECON, FLUX> Lay;
    constexpr int NV = Lay::NV;
    constexpr int S = Lay::S;
    constexpr bool LAST = KIND == KIND_RK3_2 || KIND == KIND_RK2_1;
    constexpr bool FORMS = KIND == KIND_RK3_1 || KIND == KIND_RK2_1;  // U1 formed on load
    const int lane = threadIdx.x;
    const GridDesc& gd = L.grid;
    StepState* st = L.state ? L.state + (L.subdomains ? 0 : member) : nullptr;

    R* ring = reinterpret_cast<R*>(smem);
    R* halo = ring + Lay::RING * Lay::ROW;

    const int tx = tile % gd.tiles[0];
    const int ty = tile / gd.tiles[0];
    const int x0 = gd.lo[0] + tx * Lay::TX;
    // run ty of gd.tiles[1], which split the rows evenly
    const int ny = gd.hi[1] - gd.lo[1];
    const int j0 = gd.lo[1] + int((long long)ny * ty / gd.tiles[1]);
    const int j1 = gd.lo[1] + int((long long)ny * (ty + 1) / gd.tiles[1]);
    const int rows = j1 - j0;
    const long long base = (long long)member * L.member_stride;
    const R gamma = R(P.gamma);

    R c = R(0);
    if (FORMS) {
        if (st) {
            const double dt = step_dt(st);
            if (tile == 0 && threadIdx.x == 0 && (member == 0 || !L.subdomains)) {
                st->dt = dt;
            }
            c = R(dt / st->dx[0]);
        } else {
            c = R(P.c_fixed);
        }
    } else if (KIND == KIND_RK3_2) {
        c = st ? R(st->dt / st->dx[0]) : R(P.c_fixed);
    }

    const int g = gd.ghosts;

    R wmax[2] = {R(0), R(0)};
    bool bad = false;
    long long bad_idx = 0;
    {
        // the states just outside the 32 columns, for every row of the run
#pragma unroll 1
        for (int i = lane; i < 3 * rows; i += 32) {
            const int which = i / rows;       // 0: column -1, 1: column 0, 2: column 32
            const int row = i - which * rows;
            const int x = x0 + (which == 0 ? -1 : (which == 1 ? 0 : Lay::TX));
            // every stencil cell inside the padded row; a column past the
            // region is of no use to any face, so its place may shift
            const int px = x + g + S < gd.N[0] ? x + g : gd.N[0] - 1 - S;
            StageInputFetch<R, KIND> f{&L, base + (long long)(j0 + row + g) * gd.N[0] + px, c};
            R l[NV], r[NV];
            reconstruct_f<R, NV, RECON>(f, l, r, gamma);
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                halo[which * Lay::HALO + v * kRunRows + row] = which == 0 ? r[v] : l[v];
            }
        }
        __syncwarp();
        if (lane < rows) {
            R ul[NV], ur[NV], F[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                ul[v] = halo[v * kRunRows + lane];
                ur[v] = halo[Lay::HALO + v * kRunRows + lane];
            }
            const R w = face_flux_best<R, 2, FLUX, 0>(ul, ur, gamma, F);
            if (KIND == KIND_FLUX0 && wmax[0] < w) {
                wmax[0] = w;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                halo[v * kRunRows + lane] = F[v];
            }
        }

        const int col = x0 + lane;
        const bool in_region = col < gd.hi[0];
        R* mine = ring + S + lane;       // this lane's column in slot 0
        // One row of the stage's input, as loaded (U1 is formed when the row goes
        // into the ring, a row later, so that nothing waits for its loads): this
        // lane's column x0 + lane - S, and one value of the 2 S columns after the
        // warp's, one lane per variable and column.  Columns and rows beyond the
        // grid read its last one: ordinary values whose results nobody uses.
        struct Row {
            R in[NV], un[NV], tin, tun;
        };
        const bool tail = S > 0 && lane < 2 * S * NV;
        const int tv = tail ? lane / (S > 0 ? 2 * S : 1) : 0;
        const int tk = 32 + (tail ? lane % (S > 0 ? 2 * S : 1) : 0);
        const int pa = min(x0 + lane - S + g, gd.N[0] - 1);
        const int pt = min(x0 + tk - S + g, gd.N[0] - 1);
        const R* tail_in = static_cast<const R*>(L.in[tv]);
        const R* tail_un = static_cast<const R*>(L.un[tv]);
        auto fetch_row = [&](int y, Row& r) {
            const long long first = base + (long long)min(y + g, gd.N[1] - 1) * gd.N[0];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                r.in[v] = static_cast<const R*>(L.in[v])[first + pa];
                if (FORMS) {
                    r.un[v] = static_cast<const R*>(L.un[v])[first + pa];
                }
            }
            if (tail) {
                r.tin = tail_in[first + pt];
                if (FORMS) {
                    r.tun = tail_un[first + pt];
                }
            }
        };
        auto formed = [&](R in, R un) {
            if (FORMS) {
                in = in * c;
                in = in + un;
            }
            return in;
        };
        auto store_row = [&](int slot, const Row& r) {
            R* dst = ring + slot * Lay::ROW;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                dst[v * Lay::BX + lane] = formed(r.in[v], r.un[v]);
            }
            if (tail) {
                dst[tv * Lay::BX + tk] = formed(r.tin, r.tun);
            }
        };
        auto next = [](int s) { return s + 1 == Lay::RING ? 0 : s + 1; };
        typedef RingFetch<R, Lay::RING, Lay::ROW, Lay::BX> Column;

        // rows j0-1-S .. j0-1+S into slots 0 .. 2S: the cell below the run,
        // then the first cell and the face between them
        R ry[NV], fy[NV];
        Row ahead;
#pragma unroll
        for (int k = 0; k < 2 * S + 1; ++k) {
            fetch_row(j0 - 1 - S + k, ahead);
            store_row(k, ahead);
        }
        int centre = S;                  // slot of the row reconstructed along y
        int fill = (2 * S + 1) % Lay::RING;   // slot the next row goes to
        fetch_row(j0 + S, ahead);
        __syncwarp();
        {
            R l[NV];
            reconstruct_f<R, NV, RECON>(Column{mine, centre}, l, ry, gamma);
        }
        __syncwarp();
        store_row(fill, ahead);
        fill = next(fill);
        centre = next(centre);
        fetch_row(j0 + 1 + S, ahead);
        __syncwarp();
        {
            R l[NV], r[NV];
            reconstruct_f<R, NV, RECON>(Column{mine, centre}, l, r, gamma);
            const R w = face_flux_best<R, 2, FLUX, 1>(ry, l, gamma, fy);
            if (KIND == KIND_FLUX0 && in_region && wmax[1] < w) {
                wmax[1] = w;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                ry[v] = r[v];
            }
        }

#pragma unroll 1
        for (int j = j0; j < j1; ++j) {
            // row j + 1 + S replaces the oldest; the one after it is on its way
            __syncwarp();
            store_row(fill, ahead);
            fill = next(fill);
            const int here = centre;     // slot of row j
            centre = next(centre);
            __syncwarp();
            if (j + 1 < j1) {
                fetch_row(j + 2 + S, ahead);
            }
            R un[NV];
            if (in_region) {
                load_un<R, 2, NV, KIND>(L, base, col, j, 0, un);
            }
            // this cell along x, the next one along y
            const int row = j - j0;
            R Fx[NV], Fy[NV], rn[NV], wx, wy;
            {
                R lx[NV], rx[NV], ux[NV];
                reconstruct<R, NV, RECON>(mine + here * Lay::ROW, Lay::BX, 1, lx, rx, gamma);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const R o = halo[2 * Lay::HALO + v * kRunRows + row];
                    const R n = __shfl_down_sync(0xffffffffu, lx[v], 1);
                    ux[v] = lane == 31 ? o : n;
                }
                wx = face_flux_best<R, 2, FLUX, 0>(rx, ux, gamma, Fx);
            }
            {
                R ly[NV];
                reconstruct_f<R, NV, RECON>(Column{mine, centre}, ly, rn, gamma);
                wy = face_flux_best<R, 2, FLUX, 1>(ry, ly, gamma, Fy);
            }
            if (KIND == KIND_FLUX0 && in_region) {
                wmax[0] = wmax[0] < wx ? wx : wmax[0];
                wmax[1] = wmax[1] < wy ? wy : wmax[1];
            }
            R acc[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const R o = halo[v * kRunRows + row];
                const R n = __shfl_up_sync(0xffffffffu, Fx[v], 1);
                const R tr = -Fx[v];
                const R tl = -(lane == 0 ? o : n);
                acc[v] = R(0) + (tr + (-tl));
                const R sr = -Fy[v];
                const R sl = -fy[v];
                acc[v] = acc[v] + (sr + (-sl));
                fy[v] = Fy[v];
                ry[v] = rn[v];
            }
            if (in_region) {
                R ub[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    ub[v] = mine[here * Lay::ROW + v * Lay::BX];
                }
                update_cell<R, 2, NV, KIND>(P, L, member, base, c, gamma, acc, ub, un, col, j, 0, bad,
                    bad_idx);
            }
        }
    }

    if (KIND == KIND_FLUX0) {
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const R w = warp_max(wmax[d]);
            if (lane == 0 && w > R(0)) {
                unsigned long long* dst = st ? &st->ws[d] : (L.ws_out + 3 * member + d);
                atomicMax(dst, (unsigned long long)__double_as_longlong(double(w)));
            }
        }
    }

    if (LAST && st) {
        if (bad) {
            atomicOr(&st->status, 1);
            atomicMin((unsigned long long*)&st->bad_index, (unsigned long long)bad_idx);
        }
        __syncwarp();
        if (lane == 0) {
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
__global__ void __launch_bounds__(32, rows_warps_per_sm<R>())
rows_kernel(const StageParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    walk_work(P, [&](const LevelDesc& L, int tile, int member) {
        rows_tile<R, RECON, FLUX, KIND>(P, L, tile, member, smem);
    });
}

} // namespace als
