// x / z passes of lengths without a compile-time plan (gen_engine.cuh), on tiles moved by TMA.
//
// A tile is T (a power of two) adjacent k-columns along a whole line, as in pass_tma.cuh; CTAs are
// persistent and hold three buffers: the landing buffer of the next tile and two that the stages
// alternate between.  The next tile's load is issued once the first stage has read the landing buffer,
// so it is in flight through the other stages and the store; the finished tile leaves by a TMA
// store that the next tile's first stage overlaps.  Elements past the line's end in the last box and
// past Py in the last tile are zero-filled on load and clipped on store.
//
// Mixed radices: bound by instruction issue (0.54-0.58 of the issue slots at 24 warps an SM), not by memory.
// Measured against the in-place engine of k_xz (sums over prime factors, tiles of 4096 / n columns), on
// 512 x 1140 x 270: x (1140 = 19 * 15 * 4) 2.40 -> 0.48 ms, z convolution (270) 3.80 -> 0.96 ms.
// The OTF is read straight from memory by the inverse's first stage (all its loads are issued before the
// first is used); a run-time choice of what each load and store does, element by element, took 3.42 ms there.
#pragma once
#include "gen_engine.cuh"
#include "pass_kernels.cuh"
#include "tma.cuh"

namespace pkpass {

constexpr int kGenThreads = 256;

// Elements of each of a tile's three buffers, for landing and for the stages (whole boxes: the result
// leaves from a stage buffer box by box), in multiples of 128 bytes; a launch takes the largest of its volumes.
inline int gen_buf(const GenAxis& A) { return (A.T * A.rows * A.nbox + 15) & ~15; }
inline size_t gen_smem(int buf) { return 256 + sizeof(float2) * 3 * (size_t)buf; }

struct GenKernel {   // [0]: radices up to 16, [1]: up to 31
    void (*fn[2])(const VolDesc*, const XZMaps*, const int*, int, int, int, int, int*);
};

#ifdef PK_GEN_KERNEL   // instantiated in one file
template <bool BIG>
__global__ void __launch_bounds__(kGenThreads, BIG ? 2 : 3)
    k_xzg(const VolDesc* __restrict__ descs, const XZMaps* __restrict__ maps, const int* __restrict__ prefix, int nvol,
          int axis, int mode, int buf, int* err) {
    extern __shared__ unsigned char graw[];
    unsigned char* sm = graw + ((128 - (pktma::smem_u32(graw) & 127)) & 127);
    uint64_t* bar = (uint64_t*)sm;
    sm += 128;   // keeps the tiles on 128-byte boundaries, as the TMA wants them
    const int tid = threadIdx.x;
    const int total = prefix[nvol];
    if ((int)blockIdx.x >= total) return;
    const bool conv = mode == XZ_CONV;

    struct Tile { int vol, outer, k0; };
    auto locate = [&](int g) {
        Tile t;
        t.vol = find_vol(prefix, nvol, g);
        const VolDesc& d = descs[t.vol];
        const GenAxis* A = axis == 1 ? d.ax.gen : d.az.gen;
        const int lb = g - prefix[t.vol];
        const int ctiles = (d.Py + A->T - 1) >> A->lt;
        t.outer = lb / ctiles;
        t.k0 = (lb - t.outer * ctiles) << A->lt;
        return t;
    };
    auto load = [&](const Tile& t) {   // one thread
        const VolDesc& d = descs[t.vol];
        const GenAxis* A = axis == 1 ? d.ax.gen : d.az.gen;
        pktma::mbar_expect_tx(bar, (uint32_t)(A->T * A->rows * A->nbox) * 8u);
        for (int r = 0; r < A->nbox; r++) {
            float2* dst = (float2*)sm + r * A->rows * A->T;
            if (axis == 1) pktma::tma_load_3d(dst, &maps[t.vol].s, 2 * t.k0, r * A->rows, t.outer, bar);
            else pktma::tma_load_3d(dst, &maps[t.vol].s, 2 * t.k0, t.outer, r * A->rows, bar);
        }
    };
    if (tid == 0) {
        pktma::mbar_init(bar, 1);
        pktma::fence_mbar_init();
        for (int v = 0; v < nvol; v++) pktma::tmap_acquire(&maps[v].s);
        pdl_wait();   // only this thread moves what other passes write
        load(locate(blockIdx.x));
    }
    __syncthreads();

    float2* const in = (float2*)sm;
    float2* const w0 = in + buf;
    float2* const w1 = w0 + buf;
    float2* busy = w1;   // the stage buffer that the previous tile's store reads
    uint32_t parity = 0;
    for (int g = blockIdx.x; g < total; g += gridDim.x, parity ^= 1) {
        const Tile t = locate(g);
        const VolDesc& d = descs[t.vol];
        const GenAxis* A = axis == 1 ? d.ax.gen : d.az.gen;
        const int T = A->T, lt = A->lt;
        const bool ok = pktma::mbar_wait(bar, parity);
        if (!__syncthreads_and(ok)) {
            if (tid == 0) {
                pktma::report_wait_failure(err, 1);
                pktma::bulk_wait_all();
            }
            return;
        }
        // the stages after the first write the buffer of the pending store: it has been read by then
        auto before_sync = [&] {
            if (tid == 0) pktma::bulk_wait_read_all();
        };
        auto next_load = [&] {
            if (tid == 0 && g + (int)gridDim.x < total) {
                pktma::fence_async_smem();
                load(locate(g + gridDim.x));
            }
        };
        auto nothing = [] {};
        pkgen::GenEdge e{};
        e.ncol = d.Py - t.k0;
        e.inv = mode == XZ_INV;
        e.sc = mode == XZ_FWD_SCALE ? d.xz_scale : 1.f;
        float2* const fr = busy == w0 ? w1 : w0;
        float2* res = pkgen::gen_transform<true, BIG>(A, in, fr, busy, T, lt, e, tid, kGenThreads, before_sync, next_load);
        if (conv) {
            const long long base = (axis == 1 ? (long long)t.outer * d.nx : (long long)t.outer) * d.Pp;
            e.otf = d.otf + base + t.k0;
            e.es = axis == 1 ? d.Pp : (long long)d.nx * d.Pp;
            e.conj = d.conj;
            e.inv = 1;
            res = pkgen::gen_transform<true, BIG>(A, res, res == w0 ? w1 : w0, res, T, lt, e, tid, kGenThreads, nothing, nothing);
        }
        pktma::fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            for (int r = 0; r < A->nbox; r++) {
                const float2* src = res + r * A->rows * T;
                if (axis == 1) pktma::tma_store_3d(&maps[t.vol].s, 2 * t.k0, r * A->rows, t.outer, src);
                else pktma::tma_store_3d(&maps[t.vol].s, 2 * t.k0, t.outer, r * A->rows, src);
            }
            pktma::bulk_commit();
        }
        busy = res;
    }
    if (tid == 0) pktma::bulk_wait_all();
}
#endif

}  // namespace pkpass
