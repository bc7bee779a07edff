// Launchers of the D3Q19 kernels for one storage type (included by the
// instantiation units).
#pragma once

#include <algorithm>

#include "kernels3d.cuh"
#include "ops3d.h"
#include "staged3d.cuh"
#include "tiled3d.cuh"

namespace orr {

template <class S> struct Launch3D {
    using A = typename Storage<S>::A;

    static cudaError_t step(const Geom3D& g, const void* phys, const void* src, void* dst,
                            const StepBuffers3D& b, bool smag, uint32_t block, uint32_t npt, bool chained,
                            cudaStream_t s) {
        Geom3D gg = g;
        gg.tiles_x = (g.nx + block - 1) / block;
        const auto& p = *static_cast<const Phys3D<A>*>(phys);
        const auto* in = static_cast<const S*>(src);
        auto* out = static_cast<S*>(dst);
        if constexpr (sizeof(S) == 2) {
            if (npt == 2 && pairs_ok(g, block)) {
                gg.tiles_x = (g.nx + 2 * block - 1) / (2 * block);
                const dim3 grid2(gg.tiles_x, g.ny, g.nz);
                if (smag) {
                    step3d_pair_kernel<S, true><<<grid2, block, 0, s>>>(gg, p, in, out, b);
                } else {
                    step3d_pair_kernel<S, false><<<grid2, block, 0, s>>>(gg, p, in, out, b);
                }
                return cudaGetLastError();
            }
        }
        if constexpr (sizeof(A) == 4) {
            if (step_linear(g, block)) {
                LinearOffsets3D l;
                for (int i = 0; i < d3::Q; ++i) {
                    const int64_t to = static_cast<int64_t>(i) * static_cast<int64_t>(g.cells);
                    const int64_t shift = d3::cx(i) + static_cast<int64_t>(g.nx) * d3::cy(i) +
                                          static_cast<int64_t>(g.plane) * d3::cz(i);
                    l.in[i] = static_cast<uint32_t>((to - shift) * static_cast<int64_t>(sizeof(S)));
                    l.out[i] = static_cast<uint32_t>(to * static_cast<int64_t>(sizeof(S)));
                }
                const unsigned blocks = static_cast<unsigned>((g.cells + block - 1) / block);
                return launch_step<S>(linear_kernel(smag), blocks, block, chained, s, gg, p, in, out, l, b,
                                   LinearDivs3D{fast_div(g.nx), fast_div(g.ny)});
            }
        }
        const dim3 grid(gg.tiles_x, g.ny, g.nz);
        const bool beside = b.wall_layers == kBeside;
        const auto launch = [&]<bool K>() {
            if (g.flat) {
                if constexpr (sizeof(A) == 8) {
                    if (dense_rows(g, block)) {
                        return launch_step<S>(&step3d_kernel<S, K, Walls::Halfway, 128, 5>, grid, block, chained, s, gg,
                                              p, in, out, b);
                    }
                }
                return launch_step<S>(&step3d_kernel<S, K, Walls::Halfway>, grid, block, chained, s, gg, p, in, out, b);
            }
            if (walls_listed(g, block, b.wall_count, beside)) {
                StepBuffers3D w = b;
                w.wall_layers = wall_layers(g, block, b.wall_count);
                const dim3 with_walls(gg.tiles_x, g.ny, g.nz + w.wall_layers);
                if constexpr (sizeof(S) == 2) {
                    if (roomy_walls(g) && !beside) {
                        return launch_step<S>(&step3d_kernel<S, K, Walls::Interpolated, 256, 4>, with_walls, block,
                                              chained, s, gg, p, in, out, w);
                    }
                }
                return launch_step<S>(&step3d_kernel<S, K, Walls::Interpolated>, with_walls, block, chained, s, gg, p, in,
                                   out, w);
            }
            return launch_step<S>(&step3d_kernel<S, K, Walls::General>, grid, block, chained, s, gg, p, in, out, b);
        };
        return smag ? launch.template operator()<true>() : launch.template operator()<false>();
    }

    // Layers of the grid that hold the wall list's blocks, in front of the rows'.
    static uint32_t wall_layers(const Geom3D& g, uint32_t block, uint32_t wall_count) {
        const uint64_t layer = static_cast<uint64_t>((g.nx + block - 1) / block) * g.ny * block;
        return static_cast<uint32_t>((wall_count + layer - 1) / layer);
    }

    // Whether an open lattice's interpolated walls are stepped from their list.
    // The layers share the grid's z with the rows: a lattice whose nz leaves them no
    // room takes the general node code.  So do the storages with binary32
    // arithmetic between 10,000 and 300,000 nodes, where one or two waves hold the
    // grid and the list's chain adds to the rows' (its registers spill in every
    // row), unless other lattices run beside this one (eight of 64 x 32 x 32, binary32
    // 28.7 19.8).  us per step, general and listed (40 registers), binary16: 48 x 24 x 24
    // 11.9 14.6, 64 x 32 x 32 12.0 16.6, 96 x 48 x 48 14.1 17.9; binary32 8.7 10.1, 9.6
    // 10.0, 12.0 13.6; above and below, binary32: 5 x 4 x 3 6.0 3.3, 16 x 8 x 8 with the
    // convective outlet 8.3 7.9, 112 x 56 x 56 15.6 15.2, 192 x 96 x 96 61 56.
    static bool walls_listed(const Geom3D& g, uint32_t block, uint32_t wall_count, bool beside) {
        if (!g.open || g.flat || uint64_t{g.nz} + wall_layers(g, block, wall_count) > 65535u) {
            return false;
        }
        return sizeof(A) == 8 || wall_count == 0u || beside || g.cells < 10000u || g.cells >= 300000u;
    }

    // Whether the listed form of a 2-byte storage is compiled for 64 registers
    // (4 blocks an SM) or, where more warps pay for its spills, 40 (6).  us per step
    // with 40 and 64: 24 x 12 x 12 13.6 11.4, 112 x 56 x 56 21.9 16.4, 128 x 64 x 64 22.8
    // 16.6, 144 x 72 x 72 25.9 23.1, 160 x 80 x 80 (1.0 million nodes) 29.3 28.2, with
    // sponge and convective outlet 31.5 32.4; 192 x 96 x 96 45.4 51.0.
    static bool roomy_walls(const Geom3D& g) { return sizeof(S) == 2 && g.cells < 900000u; }

    // The binary64 step waits on memory and long arithmetic with 16 warps an SM;
    // 20 at 96 registers hide more of both for some spilled values.  us per step
    // without and with: 64 x 48 x 48 14.1 13.7, 97 x 65 x 65 37.0 34.9, 128 x 64 x 64 37.9
    // 35.2, 256 x 128 x 128 239 228 (convective outlet 259 247).  Where 16 warps an SM
    // hold the lattice the spills are all that changes (64 x 32 x 32 8.1 8.4), larger
    // lattices are bound by memory (300 x 150 x 150 396 403, 337 x 193 x 193 744 766),
    // interpolated walls spill far more (337 x 193 x 193 806 827), and 24 warps at 80
    // registers are slower (256 x 128 x 128 305).
    static bool dense_rows(const Geom3D& g, uint32_t block) {
        return sizeof(A) == 8 && g.flat && block <= 128 && g.cells < 6000000u &&
               static_cast<uint64_t>((g.nx + 31) / 32) * g.ny * g.nz > 148u * 16u;
    }

    // The linear order serves flat lattices whose buffers 32-bit byte offsets
    // reach.  us per step, rows and linear:
    // The 2-byte storages gain from it (binary16 256 x 128 x 128 88 79, 337 x 193 x
    // 193 268 231) except in blocks of at most 128 threads beyond 30 million nodes
    // (128 threads, 480 x 240 x 240 567 560, 512 x 256 x 256 650 674).
    // Binary32 is bound by memory.  It gains where nx is not a multiple of 64 (66 x
    // 120 x 120 35.5 27.9, 337 x 120 x 120 134 120, 200 x 200 x 200 199 192; multiples
    // of 8 gain less and a few lose: 120 x 120 x 120 45.2 46.3, 160 59.4 60.0, 280
    // 99.3 101.0, 250 x 125 x 125 107 109), not where it is (256 x 128 x 128 102.9 104.5), and
    // not in one wave of row tiles (40 x 20 x 20 3.46 4.10, 56 x 28 x 28 4.48 5.01;
    // 72 x 36 x 36 5.25 5.33, with 64 threads 6.79 5.63; 80 x 40 x 40 7.05 5.78).
    static bool step_linear(const Geom3D& g, uint32_t block) {
        if (sizeof(A) != 4 || !g.flat || d3::Q * g.cells * sizeof(S) > 0xffffffffull) {
            return false;
        }
        return sizeof(S) == 2 ? block > 128u || g.cells < 30000000u : g.nx % 64 != 0 && g.cells >= 60000u;
    }

    static auto linear_kernel(bool smag) {
        return smag ? &step3d_linear_kernel<S, true> : &step3d_linear_kernel<S, false>;
    }

    static cudaError_t init(const Geom3D& g, const uint8_t* cls, const double* rho,
                            const double* ux, const double* uy, const double* uz, double r0,
                            double u0x, double u0y, double u0z, void* f0, cudaStream_t s) {
        const unsigned blocks = static_cast<unsigned>((g.cells + 255) / 256);
        init3d_kernel<S><<<blocks, 256, 0, s>>>(g, cls, rho, ux, uy, uz, r0, u0x, u0y, u0z,
                                                static_cast<S*>(f0));
        return cudaGetLastError();
    }

    static cudaError_t history(const Geom3D& g, const void* f, void* hist, cudaStream_t s) {
        const unsigned face = g.ny * g.nz;
        history3d_kernel<S><<<(face + 255) / 256, 256, 0, s>>>(g, static_cast<const S*>(f),
                                                               static_cast<A*>(hist));
        return cudaGetLastError();
    }

    static cudaError_t moments(const Geom3D& g, const void* phys, const uint8_t* cls,
                               const void* f, void* m, cudaStream_t s) {
        const unsigned blocks = static_cast<unsigned>((g.cells + 255) / 256);
        moments3d_kernel<S><<<blocks, 256, 0, s>>>(g, *static_cast<const Phys3D<A>*>(phys), cls,
                                                   static_cast<const S*>(f), static_cast<A*>(m));
        return cudaGetLastError();
    }

    static cudaError_t force(const Geom3D& g, const void* f, const uint32_t* lcell,
                             const uint32_t* ldir, const double* lq, uint64_t links, ForceScratch* scratch,
                             double* result, const uint32_t* status, cudaStream_t s) {
        const auto blocks = static_cast<unsigned>(
            std::clamp<uint64_t>((links + kForceThreads - 1) / kForceThreads, 1, kForceBlocks));
        force3d_kernel<S><<<blocks, kForceThreads, 0, s>>>(g, static_cast<const S*>(f), lcell, ldir, lq, links,
                                                           scratch, result, status);
        return cudaGetLastError();
    }

    static cudaError_t mass(const Geom3D& g, const uint8_t* cls, const void* f, double* out,
                            cudaStream_t s) {
        cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), s);
        if (e != cudaSuccess) {
            return e;
        }
        const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((g.cells + 255) / 256, 1184));
        mass3d_kernel<S><<<blocks, 256, 0, s>>>(g, cls, static_cast<const S*>(f), out);
        return cudaGetLastError();
    }

    // The pair step serves 2-byte storage on flat lattices with even nx, in
    // blocks of whole warps up to 128 threads.
    static bool pairs_ok(const Geom3D& g, uint32_t block) {
        return sizeof(S) == 2 && g.flat && g.nx % 2 == 0 && block % 32 == 0 && block <= 128;
    }

    static uint32_t step_grid(const Geom3D& g, uint32_t block, uint32_t npt, uint32_t wall_count) {
        if (npt == 1 && step_linear(g, block)) {
            return static_cast<uint32_t>((g.cells + block - 1) / block);
        }
        const uint32_t layers = walls_listed(g, block, wall_count, false) ? wall_layers(g, block, wall_count) : 0u;
        return (g.nx + block * npt - 1) / (block * npt) * g.ny * (g.nz + layers);
    }

    static int step_registers(const Geom3D& g, bool smag, uint32_t block, uint32_t npt, uint32_t wall_count) {
        cudaFuncAttributes a{};
        const auto registers = [&a](auto kernel) {
            return cudaFuncGetAttributes(&a, kernel) == cudaSuccess ? a.numRegs : -1;
        };
        if constexpr (sizeof(S) == 2) {
            if (npt == 2) {
                return registers(smag ? &step3d_pair_kernel<S, true> : &step3d_pair_kernel<S, false>);
            }
        }
        if constexpr (sizeof(A) == 4) {
            if (step_linear(g, block)) {
                return registers(linear_kernel(smag));
            }
        }
        if constexpr (sizeof(A) == 8) {
            if (dense_rows(g, block)) {
                return registers(smag ? &step3d_kernel<S, true, Walls::Halfway, 128, 5>
                                      : &step3d_kernel<S, false, Walls::Halfway, 128, 5>);
            }
        }
        if constexpr (sizeof(S) == 2) {
            if (walls_listed(g, block, wall_count, false) && roomy_walls(g)) {
                return registers(smag ? &step3d_kernel<S, true, Walls::Interpolated, 256, 4>
                                      : &step3d_kernel<S, false, Walls::Interpolated, 256, 4>);
            }
        }
        const auto of = [&]<Walls K>() {
            return registers(smag ? &step3d_kernel<S, true, K> : &step3d_kernel<S, false, K>);
        };
        return g.flat                                ? of.template operator()<Walls::Halfway>()
               : walls_listed(g, block, wall_count, false) ? of.template operator()<Walls::Interpolated>()
                                                     : of.template operator()<Walls::General>();
    }

    template <bool kSmag, int B, int NPT, bool kSingle> static constexpr auto staged_kernel() {
        return &step3d_staged_kernel<S, kSmag, B, NPT, kSingle>;
    }

    // Calls f.template operator()<kSmag, B, NPT>() for a supported runtime
    // shape (B 128 or 256, NPT 1 or 2); false otherwise.
    template <class F> static bool with_shape(bool smag, uint32_t block, uint32_t npt, F&& f) {
        const auto go = [&]<bool K>() {
            if (block == 256 && npt == 1) { f.template operator()<K, 256, 1>(); return true; }
            if (block == 256 && npt == 2) { f.template operator()<K, 256, 2>(); return true; }
            if (block == 128 && npt == 1) { f.template operator()<K, 128, 1>(); return true; }
            if (block == 128 && npt == 2) { f.template operator()<K, 128, 2>(); return true; }
            return false;
        };
        return smag ? go.template operator()<true>() : go.template operator()<false>();
    }

    // One lattice (host_one non-null, n == 1) travels by value, so its fields
    // are constant-bank operands; otherwise the kernel reads the device table.
    static cudaError_t staged(const void* host_one, const void* table, uint32_t n, uint64_t staged_items,
                              uint64_t direct_items, uint32_t flip, uint32_t stages, bool smag,
                              uint32_t block, uint32_t npt, uint32_t grid, uint32_t* status, cudaStream_t s) {
        if (stages == 0 || stages > kMaxStages || grid == 0 || staged_items >= (1ull << 31) ||
            direct_items >= (1ull << 31)) {
            return cudaErrorInvalidValue;
        }
        const auto* one = static_cast<const Lattice3D<A>*>(host_one);
        const auto* lats = static_cast<const Lattice3D<A>*>(table);
        const auto si = static_cast<uint32_t>(staged_items), di = static_cast<uint32_t>(direct_items);
        const bool ok = with_shape(smag, block, npt, [&]<bool K, int B, int NPT>() {
            const uint32_t smem = staged_smem_bytes<S, B * NPT>(stages);
            if (one != nullptr && n == 1) {
                staged_kernel<K, B, NPT, true>()<<<grid, kStagedThreads<B>, smem, s>>>(
                    *one, lats, n, si, di, flip, stages, status);
            } else {
                staged_kernel<K, B, NPT, false>()<<<grid, kStagedThreads<B>, smem, s>>>(
                    Lattice3D<A>{}, lats, n, si, di, flip, stages, status);
            }
        });
        return ok ? cudaGetLastError() : cudaErrorInvalidValue;
    }

    static uint32_t staged_smem(uint32_t block, uint32_t npt, uint32_t stages) {
        uint32_t bytes = 0;
        with_shape(false, block, npt, [&]<bool K, int B, int NPT>() { bytes = staged_smem_bytes<S, B * NPT>(stages); });
        return bytes;
    }

    // The kernel's dynamic shared-memory limit is raised to the device's
    // opt-in maximum (not to `smem`: solvers with different stage counts
    // share the kernel).
    template <class K> static int occupancy_of(K kernel, uint32_t threads, uint32_t smem) {
        int device = 0, optin = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (static_cast<int>(smem) > optin) {
            return 0;
        }
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        int blocks = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, static_cast<int>(threads), smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return blocks;
    }

    // Both variants (single and table) get the attribute; the occupancy is
    // the smaller of the two.
    static int staged_occupancy(bool smag, uint32_t block, uint32_t npt, uint32_t stages) {
        if (stages == 0 || stages > kMaxStages) {
            return 0;
        }
        int result = 0;
        with_shape(smag, block, npt, [&]<bool K, int B, int NPT>() {
            const uint32_t smem = staged_smem_bytes<S, B * NPT>(stages);
            const int a = occupancy_of(staged_kernel<K, B, NPT, true>(), kStagedThreads<B>, smem);
            const int b = occupancy_of(staged_kernel<K, B, NPT, false>(), kStagedThreads<B>, smem);
            result = a < b ? a : b;
        });
        return result;
    }

    static int staged_registers(bool smag, uint32_t block, uint32_t npt) {
        int regs = -1;
        with_shape(smag, block, npt, [&]<bool K, int B, int NPT>() {
            cudaFuncAttributes a{};
            if (cudaFuncGetAttributes(&a, staged_kernel<K, B, NPT, true>()) == cudaSuccess) {
                regs = a.numRegs;
            }
        });
        return regs;
    }

    // Calls f.template operator()<kSmag, R, B>() for a supported tile shape
    // (rows 8 with 512 consumers, rows 4 with 256); false otherwise.
    template <class F> static bool with_tile(bool smag, uint32_t rows, uint32_t block, F&& f) {
        const auto go = [&]<bool K>() {
            if (rows == 8 && block == 512) { f.template operator()<K, 8, 512>(); return true; }
            if (rows == 4 && block == 256) { f.template operator()<K, 4, 256>(); return true; }
            if (rows == 2 && block == 256) { f.template operator()<K, 2, 256>(); return true; }
            return false;
        };
        return smag ? go.template operator()<true>() : go.template operator()<false>();
    }

    static cudaError_t tiled(const void* host_one, const TileMaps& maps, const TileGrid& tg, uint32_t flip,
                             uint32_t stages, bool smag, uint32_t rows, uint32_t block, uint32_t grid,
                             uint32_t* status, cudaStream_t s) {
        if (stages == 0 || stages > kMaxStages || grid == 0 || host_one == nullptr) {
            return cudaErrorInvalidValue;
        }
        const auto& one = *static_cast<const Lattice3D<A>*>(host_one);
        const bool ok = with_tile(smag, rows, block, [&]<bool K, int R, int B>() {
            step3d_tiled_kernel<S, K, R, B><<<grid, kTiledThreads<B>, tiled_smem_bytes<S, R>(stages), s>>>(
                one, maps, tg, flip, stages, status);
        });
        return ok ? cudaGetLastError() : cudaErrorInvalidValue;
    }

    static int tiled_occupancy(bool smag, uint32_t rows, uint32_t block, uint32_t stages) {
        if (stages == 0 || stages > kMaxStages) {
            return 0;
        }
        int result = 0;
        with_tile(smag, rows, block, [&]<bool K, int R, int B>() {
            result = occupancy_of(&step3d_tiled_kernel<S, K, R, B>, kTiledThreads<B>,
                                  tiled_smem_bytes<S, R>(stages));
        });
        return result;
    }

    static int tiled_registers(bool smag, uint32_t rows, uint32_t block) {
        int regs = -1;
        with_tile(smag, rows, block, [&]<bool K, int R, int B>() {
            cudaFuncAttributes a{};
            if (cudaFuncGetAttributes(&a, &step3d_tiled_kernel<S, K, R, B>) == cudaSuccess) {
                regs = a.numRegs;
            }
        });
        return regs;
    }

    static cudaError_t force_batch(const void* jobs, uint32_t n, uint64_t chunks, double* partial,
                                   double* out, bool accumulate, cudaStream_t s) {
        if (n == 0) {
            return cudaSuccess;
        }
        const auto* j = static_cast<const ForceJob*>(jobs);
        if (chunks > 0) {
            force_batch_partials<S><<<static_cast<unsigned>(chunks), kForceThreads, 0, s>>>(j, n, partial);
        }
        force_batch_totals<S><<<n, kForceThreads, 0, s>>>(j, partial, out, accumulate ? 1 : 0);
        return cudaGetLastError();
    }

    static const Ops3D& table() {
        static const Ops3D ops{&step,   &init,   &history,        &moments,          &force,
                               &mass,   &step_linear, &step_grid, &step_registers, &pairs_ok, &staged, &staged_occupancy,
                               &staged_smem, &staged_registers, &tiled, &tiled_occupancy,
                               &tiled_registers, &force_batch};
        return ops;
    }
};

} // namespace orr
