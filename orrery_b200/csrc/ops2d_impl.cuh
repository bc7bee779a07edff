// Launchers of the D2Q9 kernels for one storage type.
#pragma once

#include <algorithm>

#include "kernels2d.cuh"
#include "ops2d.h"

namespace orr {

template <class S> struct Launch2D {
    using A = typename Storage<S>::A;
    static cudaError_t step(const Geom2D& g, const void* phys, const void* src, void* dst,
                            const StepBuffers2D& b, bool smag, uint32_t block, bool chained, cudaStream_t s) {
        const unsigned blocks = static_cast<unsigned>((g.cells + block - 1) / block);
        const auto& p = *static_cast<const Phys2D<A>*>(phys);
        const auto launch = [&]<class O>() {
            LinearOffsets2D<O> l;
            for (int i = 0; i < d2::Q; ++i) {
                const int64_t to = static_cast<int64_t>(i) * static_cast<int64_t>(g.cells);
                const int64_t shift = d2::cx(i) + static_cast<int64_t>(g.nx) * d2::cy(i);
                l.in[i] = static_cast<O>((to - shift) * static_cast<int64_t>(sizeof(S)));
                l.out[i] = static_cast<O>(to * static_cast<int64_t>(sizeof(S)));
            }
            l.last = static_cast<O>((d2::Q * g.cells - 1) * sizeof(S));
            const auto kernel = smag ? &step2d_kernel<S, true, O> : &step2d_kernel<S, false, O>;
            return launch_step<S>(kernel, blocks, block, chained, s, g, p, static_cast<const S*>(src),
                               static_cast<S*>(dst), l, b, fast_div(g.nx));
        };
        // Past the buffer's end by at most a row before it is held: the sums
        // must not wrap.
        if ((d2::Q * g.cells + g.nx) * sizeof(S) <= 0xffffffffull) {
            return launch.template operator()<uint32_t>();
        }
        return launch.template operator()<uint64_t>();
    }

    static cudaError_t init(const Geom2D& g, const uint8_t* cls, const double* rho,
                            const double* ux, const double* uy, double u0x, double u0y, void* f0,
                            cudaStream_t s) {
        const unsigned blocks = static_cast<unsigned>((g.cells + 255) / 256);
        init2d_kernel<S><<<blocks, 256, 0, s>>>(g, cls, rho, ux, uy, u0x, u0y, static_cast<S*>(f0));
        return cudaGetLastError();
    }

    static cudaError_t history(const Geom2D& g, const void* f, void* hist, cudaStream_t s) {
        history2d_kernel<S><<<(g.ny + 255) / 256, 256, 0, s>>>(g, static_cast<const S*>(f),
                                                               static_cast<A*>(hist));
        return cudaGetLastError();
    }

    static cudaError_t moments(const Geom2D& g, const void* phys, const uint8_t* cls,
                               const void* f, void* m, cudaStream_t s) {
        const unsigned blocks = static_cast<unsigned>((g.cells + 255) / 256);
        moments2d_kernel<S><<<blocks, 256, 0, s>>>(g, *static_cast<const Phys2D<A>*>(phys), cls,
                                                   static_cast<const S*>(f), static_cast<A*>(m));
        return cudaGetLastError();
    }

    static cudaError_t force(const Geom2D& g, const void* f, const uint32_t* lcell,
                             const uint32_t* ldir, uint64_t links, ForceScratch* scratch, double* result,
                             cudaStream_t s) {
        const auto blocks = static_cast<unsigned>(
            std::clamp<uint64_t>((links + kForceThreads - 1) / kForceThreads, 1, kForceBlocks));
        force2d_kernel<S><<<blocks, kForceThreads, 0, s>>>(g, static_cast<const S*>(f), lcell, ldir, links, scratch,
                                                           result);
        return cudaGetLastError();
    }

    static cudaError_t mass(const Geom2D& g, const uint8_t* cls, const void* f, double* out,
                            cudaStream_t s) {
        cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), s);
        if (e != cudaSuccess) {
            return e;
        }
        const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((g.cells + 255) / 256, 1184));
        mass2d_kernel<S><<<blocks, 256, 0, s>>>(g, cls, static_cast<const S*>(f), out);
        return cudaGetLastError();
    }

    static const Ops2D& table() {
        static const Ops2D ops{&step, &init, &history, &moments, &force, &mass};
        return ops;
    }
};

} // namespace orr
