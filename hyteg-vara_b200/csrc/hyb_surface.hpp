// The interface passes of a multicolour SOR sweep as one launch (hyb_surface.cu).
#pragma once

#include <cuda_runtime.h>

#include "hyb_device.cuh"

namespace hyb {

// Rows [ja, jb) of the interior of macro-face f (row j holds its points (i, j))
struct FaceTile
{
   int32_t f, ja, jb;
};

// Tiles of the inner macro-faces of a level, dealt to blocks, and the edge and vertex DoFs of
// each SOR colour
struct SurfaceDev
{
   int             nBlocks;
   int             most;    // points of one block's tiles at most, with their rows' neighbours
   int             tiles;   // tiles of one block at most
   const FaceTile* tile;
   const int32_t*  tileOff; // [nBlocks + 1]
   const int32_t*  list;    // the level's surface-DoF lists by colour
   int             m;       // colours
   int             off[16][3]; // per colour: offset in list, #vertex, #edge DoFs
};

constexpr int kSurfaceMaxColours = 16;
constexpr int kSurfaceMaxTiles   = 16; // tiles a block takes at most

// shared memory of a launch in a value type of elem bytes, and the most a block may take
size_t           surfaceSmem( const SurfaceDev& sf, int elem );
constexpr size_t kSurfaceMaxSmem = 200 * 1024;

// Sets up the launch on the current device (the opt-in to its shared memory is kept per device:
// every storage that has tiles calls this when it is built) and tells whether the device can run
// it: with room for the whole grid, and not under MPS, where a cooperative launch is not allowed
// in the body of a graph's loop, as the device-iterated solves have it.
bool surfacePrepare( const SurfaceDev& sf );

// All interface colours of one sweep (in the order 0 .. m-1, backwards: m-1 .. 0), for the
// DoFs on Inner | Neumann. A cooperative launch; cudaErrorCooperativeLaunchTooLarge, captured or
// not and with nothing launched, when the stream's SMs (a green context's part of the device)
// cannot hold the grid.
template < typename T >
cudaError_t launchSurfaceSor( const TopoDev& tp, const LevelDev& lv, const SurfaceDev& sf, const OpDev< T >& op, T* u,
                              const T* rhs, T relax, bool backwards, cudaStream_t stream );

} // namespace hyb
