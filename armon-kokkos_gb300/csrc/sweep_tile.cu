// sweep_tile.cu -- the tile form of the axis pass (sweep_tile.cuh) for both storage types.
// Built with --fmad=false and IEEE division / square root, like the marches.
#define ARMON_SFP_CALLS
#include "launch.h"
#include "sweep_tile.cuh"

namespace armon {
namespace {

template <class T, int S, int P>
cudaError_t launch_tile_one(const SweepArgs<T>& a, TileCtl* ctl, bool last, int grid, cudaStream_t st)
{
    if (a.reuse && (a.geom[0].tile_scan || a.geom[1].tile_scan))
        tile_kernel<T, S, P, true><<<grid, kTileThreads, 0, st>>>(a, ctl, last ? 1 : 0);
    else
        tile_kernel<T, S, P, false><<<grid, kTileThreads, 0, st>>>(a, ctl, last ? 1 : 0);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_tile_t(const SweepArgs<T>& a, TileCtl* ctl, int scheme, int proj, bool last, int grid, cudaStream_t st)
{
    if (scheme == 1)
        return proj == 2 ? launch_tile_one<T, 1, 2>(a, ctl, last, grid, st) : launch_tile_one<T, 1, 1>(a, ctl, last, grid, st);
    return proj == 2 ? launch_tile_one<T, 0, 2>(a, ctl, last, grid, st) : launch_tile_one<T, 0, 1>(a, ctl, last, grid, st);
}

template <class T>
int tile_blocks_t(int scheme, int proj)
{
    int n = 0;
    cudaError_t e;
    if (scheme == 1)
        e = proj == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_kernel<T, 1, 2, true>, kTileThreads, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_kernel<T, 1, 1, true>, kTileThreads, 0);
    else
        e = proj == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_kernel<T, 0, 2, true>, kTileThreads, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_kernel<T, 0, 1, true>, kTileThreads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

template <class T>
cudaError_t launch_tile_batch_t(const SweepArgs<T>* doms, const int* first, const int* units, const int* rest, int nrest,
                                uint32_t* tickets, int ndom, int pass, TileCtl* ctl, int scheme, int proj, bool last, int grid, cudaStream_t st)
{
#define ARMON_TB(S, P) \
    tile_batch_kernel<T, S, P><<<grid, kTileThreads, 0, st>>>(doms, first, units, rest, nrest, tickets, ndom, pass, ctl, \
                                                         last ? 1 : 0)
    if (scheme == 1) {
        if (proj == 2) ARMON_TB(1, 2); else ARMON_TB(1, 1);
    } else {
        if (proj == 2) ARMON_TB(0, 2); else ARMON_TB(0, 1);
    }
#undef ARMON_TB
    return cudaGetLastError();
}

template <class T>
int tile_batch_blocks_t(int scheme, int proj)
{
    int n = 0;
    cudaError_t e;
    if (scheme == 1)
        e = proj == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_batch_kernel<T, 1, 2>, kTileThreads, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_batch_kernel<T, 1, 1>, kTileThreads, 0);
    else
        e = proj == 2 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_batch_kernel<T, 0, 2>, kTileThreads, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, tile_batch_kernel<T, 0, 1>, kTileThreads, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

}  // namespace

cudaError_t launch_sweep_tile(const SweepArgs<double>& a, TileCtl* ctl, int scheme, int proj, bool last, int grid,
                              cudaStream_t st)
{
    return launch_tile_t<double>(a, ctl, scheme, proj, last, grid, st);
}

cudaError_t launch_sweep_tile(const SweepArgs<float>& a, TileCtl* ctl, int scheme, int proj, bool last, int grid,
                              cudaStream_t st)
{
    return launch_tile_t<float>(a, ctl, scheme, proj, last, grid, st);
}

cudaError_t launch_sweep_tile_batch(const SweepArgs<double>* doms, const int* first, const int* units, const int* rest,
                                    int nrest, uint32_t* tickets, int ndom, int pass, TileCtl* ctl, int scheme, int proj, bool last, int grid,
                                    cudaStream_t st)
{
    return launch_tile_batch_t<double>(doms, first, units, rest, nrest, tickets, ndom, pass, ctl, scheme, proj, last, grid, st);
}

cudaError_t launch_sweep_tile_batch(const SweepArgs<float>* doms, const int* first, const int* units, const int* rest,
                                    int nrest, uint32_t* tickets, int ndom, int pass, TileCtl* ctl, int scheme, int proj, bool last, int grid,
                                    cudaStream_t st)
{
    return launch_tile_batch_t<float>(doms, first, units, rest, nrest, tickets, ndom, pass, ctl, scheme, proj, last, grid, st);
}

int sweep_tile_batch_blocks_per_sm(bool fp32, int scheme, int proj)
{
    return fp32 ? tile_batch_blocks_t<float>(scheme, proj) : tile_batch_blocks_t<double>(scheme, proj);
}

int sweep_tile_blocks_per_sm(bool fp32, int scheme, int proj)
{
    return fp32 ? tile_blocks_t<float>(scheme, proj) : tile_blocks_t<double>(scheme, proj);
}

}  // namespace armon
