// Per-storage launch table of the D3Q19 kernels.  The kernels are
// instantiated in kernels_f32.cu, kernels_f16.cu, kernels_bf16.cu and
// kernels_f64.cu (double, built without FMA contraction); the solver
// reaches them only through this table.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "tiles.h"

namespace orr {

struct Geom3D;
struct StepBuffers3D;
struct ForceScratch;

// Threads per block of the linear-order step where the caller names none: 256
// from 5.5 million nodes on, 128 below.  us per step with 128 and 256, binary16
// and binary32, convective outlet: 112 x 56 x 56 13.2 13.9, 11.1 12.1; 240 x 120 x
// 120 68.5 70.0, 87.5 88.3; 272 x 136 x 136 (5.0 million) 97.4 97.5, 124.9 125.2;
// 300 x 150 x 150 (6.8 million) 135.7 127.8, 165.6 165.4; 400 x 200 x 200 340 293,
// 382 379; 512 x 256 x 256 692 589 (binary16).
inline uint32_t linear_block(uint64_t cells) { return cells >= 5500000u ? 256u : 128u; }

// Block of a batch member's row step: the schedule's, or the member's own where it
// runs in linear order and nobody named one.
inline uint32_t row_block(uint32_t block, bool named, bool linear, uint64_t cells) {
    return linear && !named ? linear_block(cells) : block;
}

// Whether the binary64 row step of an open lattice takes one-warp blocks where
// the caller names none.  Its blocks are limited by registers (16 or 20 warps an
// SM; the figures are with 16), and the warps of a 128-node tile beyond the row's
// end keep theirs until the tile is done: one-warp blocks have none.  They start
// later, so tiles stay where a wave holds them all (4 an SM, 148 SMs) or the rows
// are short and leave one warp idle.  us per step with 128 and 32 nodes, halfway
// walls: nx 64 10.3 8.1, 160 85.0 76.3, 200 158 145, 300 471 426, 337 634 590 (ny =
// nz = nx / 2); not taken: 40 6.3 6.6, 80 14.7 14.7 (interpolated walls 14.9 15.2),
// 97 21.8 24.0, 128 x 64 x 64 38.3 39.3.  The line stands with the 96-register form
// too (5 tiles an SM): 300 x 14 x 14 (588 tiles) 6.9 7.2, 160 x 18 x 18 (648) 8.7 7.0, 300 x
// 15 x 15 (675) 8.4 7.3, 300 x 16 x 16 (768) 8.5 7.7.
inline bool one_warp_rows(uint64_t nx, uint64_t ny, uint64_t nz) {
    const uint64_t idle = (4u - (nx + 31u) / 32u % 4u) % 4u;   // warps of the last tile
    return (nx > 128u ? idle > 0u : idle >= 2u) && (nx + 127u) / 128u * ny * nz > 4u * 148u;
}

struct Ops3D {
    // One fused step src -> dst (one launch).  `phys` points at a Phys3D of
    // the storage's arithmetic type; `block` is the block width (threads
    // along x of a row, or of a linear tile where step_linear says so); npt 2
    // takes the pair step (two neighbouring nodes per thread) where pairs_ok
    // allows it, the one-node step otherwise.  chained: the launch before it on
    // the stream is the same solver's step (the one-node steps overlap its end).
    cudaError_t (*step)(const Geom3D& g, const void* phys, const void* src, void* dst,
                        const StepBuffers3D& b, bool smag, uint32_t block, uint32_t npt, bool chained,
                        cudaStream_t s);
    // Equilibrium initialisation of a population buffer; rho..uz may be
    // device arrays (all non-null) or null for the uniform state (r0, u0).
    cudaError_t (*init)(const Geom3D& g, const uint8_t* cls, const double* rho, const double* ux,
                        const double* uy, const double* uz, double r0, double u0x, double u0y,
                        double u0z, void* f0, cudaStream_t s);
    cudaError_t (*history)(const Geom3D& g, const void* f, void* hist, cudaStream_t s);
    cudaError_t (*moments)(const Geom3D& g, const void* phys, const uint8_t* cls, const void* f,
                           void* m, cudaStream_t s);
    // Force and moment into `result`, 6 values in pinned host memory, and the
    // word at `status` (may be null) after them; `scratch` is the solver's.
    cudaError_t (*force)(const Geom3D& g, const void* f, const uint32_t* lcell,
                         const uint32_t* ldir, const double* lq, uint64_t links, ForceScratch* scratch,
                         double* result, const uint32_t* status, cudaStream_t s);
    cudaError_t (*mass)(const Geom3D& g, const uint8_t* cls, const void* f, double* out,
                        cudaStream_t s);
    // Whether the one-node step of lattice g in blocks of `block` threads runs in
    // linear order.
    bool (*step_linear)(const Geom3D& g, uint32_t block);
    // Blocks of lattice g's step kernel (wall_count: StepBuffers3D's).
    uint32_t (*step_grid)(const Geom3D& g, uint32_t block, uint32_t npt, uint32_t wall_count);
    // Registers per thread of lattice g's step kernel (wall_count: StepBuffers3D's).
    int (*step_registers)(const Geom3D& g, bool smag, uint32_t block, uint32_t npt, uint32_t wall_count);
    // Whether the pair step serves lattice g with blocks of `block` threads
    // (2-byte storage, periodic or free-slip sides and halfway walls, even nx,
    // whole warps up to 128 threads).
    bool (*pairs_ok)(const Geom3D& g, uint32_t block);
    // Persistent step over a device table of n Lattice3D entries of the
    // storage's arithmetic type (staged3d.cuh): `grid` CTAs of `block`
    // consumer threads (128 or 256) plus a producer warp, spans of
    // block * npt nodes (npt 1 or 2), `stages` pipeline stages, source buffer
    // f[parity ^ flip] of every lattice.  With n == 1 and `host_one` (a host
    // copy of the entry) the entry is passed by value.
    cudaError_t (*staged)(const void* host_one, const void* table, uint32_t n, uint64_t staged_items,
                          uint64_t direct_items, uint32_t flip, uint32_t stages, bool smag,
                          uint32_t block, uint32_t npt, uint32_t grid, uint32_t* status, cudaStream_t s);
    // Resident CTAs per SM of the persistent step for (smag, block, npt,
    // stages), after raising the kernel's dynamic shared-memory limit; 0 if
    // it cannot launch.
    int (*staged_occupancy)(bool smag, uint32_t block, uint32_t npt, uint32_t stages);
    // Dynamic shared memory of the persistent step, bytes.
    uint32_t (*staged_smem)(uint32_t block, uint32_t npt, uint32_t stages);
    // Registers per thread of the persistent step.
    int (*staged_registers)(bool smag, uint32_t block, uint32_t npt);
    // Persistent tiled step of one flat lattice (tiled3d.cuh): `host_one` a
    // host copy of its Lattice3D entry (passed by value), `maps` its tensor
    // maps, `tg` its tile numbering for tiles of `rows` rows and `block`
    // consumer threads (rows 8 with 512 threads, or rows 4 with 256), `grid`
    // CTAs, `stages` pipeline stages, source buffer f[parity ^ flip].
    cudaError_t (*tiled)(const void* host_one, const TileMaps& maps, const TileGrid& tg, uint32_t flip,
                         uint32_t stages, bool smag, uint32_t rows, uint32_t block, uint32_t grid, uint32_t* status,
                         cudaStream_t s);
    // Resident CTAs per SM of the tiled step (0: cannot launch) and its
    // registers per thread.
    int (*tiled_occupancy)(bool smag, uint32_t rows, uint32_t block, uint32_t stages);
    int (*tiled_registers)(bool smag, uint32_t rows, uint32_t block);
    // Momentum exchange of n lattices (device table of ForceJob, kernels3d.cuh)
    // summed in a fixed order: pass 1 over `chunks` link chunks into
    // `partial` (6 doubles per chunk), pass 2 into out[6 l ..] (added to it
    // when `accumulate`).
    cudaError_t (*force_batch)(const void* jobs, uint32_t n, uint64_t chunks, double* partial,
                               double* out, bool accumulate, cudaStream_t s);
};

const Ops3D& ops3d_f32();
const Ops3D& ops3d_f16();
const Ops3D& ops3d_bf16();
const Ops3D& ops3d_f64();

} // namespace orr
