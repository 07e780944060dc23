// The interface passes of a multicolour SOR sweep (macro-faces, -edges, -vertices) as one
// cooperative launch.
#include "hyb_surface.hpp"

#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>
#include <cuda.h>

#include "hyb_surface_dofs.cuh"

namespace hyb {

// ---------------------------------------------------------------------------
// One launch per colour gathers, for every face DoF, the values around it in both adjacent
// cells: about 24 reads of which most hit a sector of their own (a face x = 0 or
// x + y + z = N of a cell has one point per row of the slab), six colours a sweep, bound by
// the sectors and their latency and not by their bytes.
//
// The neighbours of a face point off its face are cell-interior points, which the interface
// passes do not change, unless the point lies next to an edge of the face. So a block keeps
// whole macro-faces (or ranges of their rows) in shared memory through all colours: the
// points' values u, and for each point away from the edges c0 = rhs - sum of the weights
// times the values off the face, formed once. A colour pass then reads shared memory alone
// and writes both replicas. The points next to an edge couple to other faces' points;
// they, the edges and the vertices take the general rows on the slabs (read through L2, as
// other blocks write them). Blocks exchange values through the slabs, a grid barrier per
// colour apart.
//
// One sweep's interfaces, six launches against this one: FP64 at level 7 on 48 cells 134 and
// 100 us, FP32 at level 6 on 384 cells 165 and 130. A quarter of it is the forming of c0, the
// rest the points next to an edge (a chain of L2 reads a colour) and the barriers. Bringing
// the layers behind the face into shared memory first, a sector per value instead of four,
// took 107 and 138 us: the two extra phases cost more than the sectors.
// ---------------------------------------------------------------------------
constexpr int kSurfaceThreads = 768;

// the points of an adjacent cell as an affine map of the face's coordinates: x = x0 + xi i + xj j
struct FaceSide
{
   int cell;
   int x0, xi, xj, y0, yi, yj, z0, zi, zj;
   int dq[4]; // offsets of the neighbours off the face, into the cell: (dx + 1) | (dy + 1) << 2 | (dz + 1) << 4
};

template < typename T >
struct TileDev
{
   int      ja, jb;      // rows
   int      first, count; // face index of the first point, number of points
   int      base;         // shared index of the first point
   int      h0, h1;       // face indices [h0, h1) held: the tile's rows and one on either side
   FaceSide side[2];
   T        wOff[2][4];
   T        wIn[6]; // in-face neighbours (1,0) (-1,0) (0,1) (0,-1) (1,-1) (-1,1)
   T        diag;
   int      lab[3];
};

// values read through L2: other blocks of the launch write them
template < typename T >
struct L2Ptr
{
   const T* p;
   __device__ __forceinline__ T operator[]( size_t i ) const { return __ldcg( p + i ); }
};

__device__ __forceinline__ int faceIndex( int N, int i, int j ) { return ( j - 1 ) * ( N - 1 ) - ( j - 1 ) * j / 2 + i - 1; }

template < typename T >
__global__ void __launch_bounds__( kSurfaceThreads, 1 )
    k_surface_sor( TopoDev tp, LevelDev lv, const __grid_constant__ SurfaceDev sf, OpDev< T > op, T* u,
                   const T* __restrict__ rhs, T relax, int backwards )
{
   extern __shared__ __align__( 16 ) unsigned char smem[];
   T* const        su    = reinterpret_cast< T* >( smem );            // values of the held points
   T* const        sc    = su + sf.most;                              // c0 of the points away from the edges
   uint16_t* const deep  = reinterpret_cast< uint16_t* >( sc + sf.most ); // points by tile and colour, i | j << 7
   __shared__ TileDev< T > tiles[kSurfaceMaxTiles];
   __shared__ int          cnt[2][kSurfaceMaxTiles][kSurfaceMaxColours + 1]; // [away from / next to an edge]: list ends
   namespace cg = cooperative_groups;
   const cg::grid_group grid = cg::this_grid();
   const int N = lv.N, W = lv.W, nT = sf.tileOff[blockIdx.x + 1] - sf.tileOff[blockIdx.x];
   const int tid = threadIdx.x;

   for ( int i = tid; i < 2 * kSurfaceMaxTiles * ( kSurfaceMaxColours + 1 ); i += kSurfaceThreads )
      ( &cnt[0][0][0] )[i] = 0;
   // a warp describes each tile, a lane each stencil offset
   if ( tid >> 5 < nT )
   {
      TileDev< T >&  t    = tiles[tid >> 5];
      const FaceTile ft   = sf.tile[sf.tileOff[blockIdx.x] + ( tid >> 5 )];
      const int      lane = tid & 31;
      if ( lane < 6 )
         t.wIn[lane] = 0;
      if ( lane == 0 )
      {
         t.ja    = ft.ja;
         t.jb    = ft.jb;
         t.first = faceIndex( N, 1, ft.ja );
         t.count = faceIndex( N, 1, ft.jb ) - t.first;
         t.h0    = faceIndex( N, 1, max( ft.ja - 1, 1 ) );
         t.h1    = faceIndex( N, 1, min( ft.jb + 1, N - 1 ) );
         t.diag  = 0;
      }
      __syncwarp();
      for ( int s = 0; s < 2; ++s )
      {
         const int32_t packed = embAt( tp, 2, ft.f, s );
         const int     cell   = packed & 0xFFFFFF;
         FaceSide&     fs     = t.side[s];
         const int k0 = ( packed >> 24 ) & 3, k1 = ( packed >> 26 ) & 3, k2 = ( packed >> 28 ) & 3, o = 6 - k0 - k1 - k2;
         const int q  = min( lane, 14 );
         const T   w  = __ldg( op.st + ( size_t( cell ) * 16 + ( 1 << o ) ) * 15 + q );
         const int dx = offX( q ), dy = offY( q ), dz = offZ( q );
         auto      db = [&]( int k ) { return k == 0 ? -dx - dy - dz : k == 1 ? dx : k == 2 ? dy : dz; };
         // four offsets lead into the cell, six stay on the face
         const bool     into = lane >= 1 && lane < 15 && db( o ) == 1;
         const unsigned m    = __ballot_sync( 0xffffffffu, into );
         if ( into )
         {
            const int n  = __popc( m & ( ( 1u << lane ) - 1 ) );
            fs.dq[n]     = ( dx + 1 ) | ( dy + 1 ) << 2 | ( dz + 1 ) << 4;
            t.wOff[s][n] = w;
         }
         else if ( lane >= 1 && lane < 15 && db( o ) == 0 )
         {
            const int di = db( k1 ), dj = db( k2 );
            t.wIn[dj == 0 ? ( di > 0 ? 0 : 1 ) : di == 0 ? ( dj > 0 ? 2 : 3 ) : ( di > 0 ? 4 : 5 )] += w;
         }
         if ( lane == 0 )
         {
            t.diag += w;
            fs.cell = cell;
            // barycentric coordinate k of the face point: N - i - j on k0, i on k1, j on k2
            auto c0 = [&]( int k ) { return k == k0 ? N : 0; };
            auto ci = [&]( int k ) { return k == k0 ? -1 : k == k1 ? 1 : 0; };
            auto cj = [&]( int k ) { return k == k0 ? -1 : k == k2 ? 1 : 0; };
            fs.x0 = c0( 1 ), fs.xi = ci( 1 ), fs.xj = cj( 1 );
            fs.y0 = c0( 2 ), fs.yi = ci( 2 ), fs.yj = cj( 2 );
            fs.z0 = c0( 3 ), fs.zi = ci( 3 ), fs.zj = cj( 3 );
            if ( s == 0 )
            {
               const int8_t* l = tp.labels + 4 * cell;
               t.lab[0] = l[k0], t.lab[1] = l[k1], t.lab[2] = l[k2];
            }
         }
         __syncwarp(); // the other side adds to the same weights
      }
   }
   __syncthreads();
   if ( tid == 0 )
   {
      int base = 0;
      for ( int i = 0; i < nT; ++i )
      {
         tiles[i].base = base + tiles[i].first - tiles[i].h0;
         base += tiles[i].h1 - tiles[i].h0;
      }
   }
   __syncthreads();
   auto coords = [&]( int idx, int& i, int& j ) {
      // row of a face index, counted from the short rows at the end
      const int rr = lv.nIntFace - 1 - idx;
      int       k  = int( ( sqrtf( 8.0f * float( rr ) + 1.0f ) - 1.0f ) * 0.5f );
      while ( ( k + 1 ) * ( k + 2 ) / 2 <= rr )
         ++k;
      while ( k * ( k + 1 ) / 2 > rr )
         --k;
      i = ( k + 1 ) * ( k + 2 ) / 2 - rr;
      j = N - 2 - k;
   };
   auto colourAt = [&]( const TileDev< T >& t, int i, int j ) {
      return ( t.lab[0] * ( N - i - j ) + t.lab[1] * i + t.lab[2] * j ) % sf.m;
   };
   auto slabAt = [&]( const FaceSide& fs, int i, int j, int dq ) {
      const int x = fs.x0 + fs.xi * i + fs.xj * j + ( dq & 3 ) - 1, y = fs.y0 + fs.yi * i + fs.yj * j + ( ( dq >> 2 ) & 3 ) - 1,
                z = fs.z0 + fs.zi * i + fs.zj * j + ( dq >> 4 ) - 1;
      return size_t( fs.cell ) * lv.stride + sidx( W, x, y, z );
   };
   constexpr int kSelf = 1 | 1 << 2 | 1 << 4; // the offset (0, 0, 0)
   auto          isDeep = [&]( int i, int j ) { return i >= 2 && j >= 2 && N - i - j >= 2; };
   // count the points of every colour, then lay out the lists, then fill them and form c0
   for ( int n = 0; n < nT; ++n )
   {
      const TileDev< T >& t = tiles[n];
      for ( int idx = tid; idx < t.count; idx += kSurfaceThreads )
      {
         int i, j;
         coords( t.first + idx, i, j );
         atomicAdd( &cnt[isDeep( i, j ) ? 0 : 1][n][colourAt( t, i, j ) + 1], 1 );
      }
   }
   __syncthreads();
   if ( tid < nT )
   {
      // list of tile n: away from the edges by colour, then next to the edges by colour
      int at = tiles[tid].base;
      for ( int k = 0; k < 2; ++k )
      {
         cnt[k][tid][0] = at;
         for ( int c = 1; c <= sf.m; ++c )
            cnt[k][tid][c] = at += cnt[k][tid][c];
      }
   }
   __syncthreads();
   // (the fill takes each colour's end down to its start and leaves the starts in place: the
   // end of colour c is the start of colour c + 1, in the next slot)
   for ( int n = 0; n < nT; ++n )
   {
      const TileDev< T >& t = tiles[n];
      for ( int idx = t.h0 + tid; idx < t.h1; idx += kSurfaceThreads )
      {
         int i, j;
         coords( idx, i, j );
         const size_t r0  = slabAt( t.side[0], i, j, kSelf );
         const int    si  = t.base + idx - t.first;
         const bool   own = j >= t.ja && j < t.jb, d = own && isDeep( i, j );
         const T      ui  = u[r0];
         if ( d )
         {
            // one value and right-hand side and the eight neighbours off the face, in flight together
            T       v[8];
            const T bi = rhs[r0];
#pragma unroll
            for ( int q = 0; q < 8; ++q )
               v[q] = u[slabAt( t.side[q >> 2], i, j, t.side[q >> 2].dq[q & 3] )];
            T c0 = 0, c1 = 0;
#pragma unroll
            for ( int q = 0; q < 4; ++q )
            {
               c0 += t.wOff[0][q] * v[q];
               c1 += t.wOff[1][q] * v[q + 4];
            }
            sc[si] = bi - ( c0 + c1 );
         }
         su[si] = ui;
         if ( !own )
            continue;
         deep[atomicSub( &cnt[d ? 0 : 1][n][colourAt( t, i, j ) + 1], 1 ) - 1] = uint16_t( i | j << 7 );
      }
   }
   __syncthreads();
   // now cnt[.][n][c + 1] is the first entry of colour c; its end is the next colour's first
   auto listEnd = [&]( int k, int n, int c ) {
      return c + 1 < sf.m ? cnt[k][n][c + 2] : k == 0 ? cnt[1][n][1] : tiles[n].base + tiles[n].count;
   };

   for ( int step = 0; step < sf.m; ++step )
   {
      const int c = backwards ? sf.m - 1 - step : step;
      // rows at the tiles' borders: the neighbouring tile's points of the last colour
      if ( step > 0 )
      {
         const int cp = backwards ? c + 1 : c - 1;
         for ( int n = 0; n < nT; ++n )
         {
            const TileDev< T >& t  = tiles[n];
            const int           nb = t.first - t.h0, na = t.h1 - ( t.first + t.count );
            for ( int k = tid; k < nb + na; k += kSurfaceThreads )
            {
               const int idx = k < nb ? t.h0 + k : t.first + t.count + ( k - nb );
               int       i, j;
               coords( idx, i, j );
               if ( colourAt( t, i, j ) == cp )
                  su[t.base + idx - t.first] = __ldcg( u + slabAt( t.side[0], i, j, kSelf ) );
            }
         }
         __syncthreads();
      }
      // vertices and edges: lane groups over the whole grid; points next to an edge: lane
      // pairs of the block that holds them
      {
         const int32_t*  list = sf.list + sf.off[c][0];
         const BdryLists bl{ list, list + sf.off[c][1], nullptr, sf.off[c][1], sf.off[c][2], 0 };
         const long      total = bdryLaneCount( bl.nv, bl.ne, 0 );
         // consecutive warps of the lists go to different blocks
         const long step_ = long( gridDim.x ) * kSurfaceThreads;
         for ( long gt = ( long( tid >> 5 ) * gridDim.x + blockIdx.x ) * 32 + ( tid & 31 ); gt - ( tid & 31 ) < total; gt += step_ )
         {
            const LaneTask  tk     = laneTask( tp, lv, bl, gt );
            const BdryPoint p      = decodeBdry( tp, lv, tk.t );
            const bool      active = tk.valid && ( primBc( tp, p.kind, p.prim ) & ( 1 | 4 ) );
            T               diag = 0, off = 0, own = 0, b = 0;
            if ( active )
            {
               // read before the sums: their full-warp shuffles come between every lane's read
               // of the first replica and the write of it
               const size_t r0 = bdryReplica< T >( tp, lv, p, 0 );
               own             = __ldcg( u + r0 );
               b               = rhs[r0];
               const int ne    = numEmb( tp, p.kind, p.prim );
               for ( int e = tk.sub; e < ne; e += tk.G )
               {
                  int cell, x, y, z;
                  embeddingCoords( embAt( tp, p.kind, p.prim, e ), p.kind, N, p.i, p.j, cell, x, y, z );
                  partialRow< T, 0, kRowAll >( op, L2Ptr< T >{ u + size_t( cell ) * lv.stride }, cell, W, x, y, z, diag, off );
               }
            }
            diag = groupSum( diag, tk.G );
            off  = groupSum( off, tk.G );
            if ( !active )
               continue;
            const T v = ( T( 1 ) - relax ) * own + relax * ( b - off ) / diag;
            bdryWriteGroup( tp, lv, p, tk, u, v );
         }
      }
      // (warps run whole, the pair sums are full-warp shuffles; a tile's list starts at the warp
      // where the previous tile's ended, so that the tiles' short lists run side by side)
      int shift = 0;
      for ( int n = 0; n < nT; ++n )
      {
         const TileDev< T >& t  = tiles[n];
         const int           a  = cnt[1][n][c + 1], lanes = 2 * ( listEnd( 1, n, c ) - a );
         const int           me = ( tid + kSurfaceThreads - shift ) % kSurfaceThreads;
         shift                  = ( shift + ( lanes + 31 ) / 32 * 32 ) % kSurfaceThreads;
         for ( int k = me; k - ( me & 31 ) < lanes; k += kSurfaceThreads )
         {
            const bool valid = k < lanes;
            int        si = 0;
            T          diag = 0, off = 0, bi = 0;
            size_t     r = 0;
            if ( valid )
            {
               const int       ij = deep[a + ( k >> 1 )], i = ij & 127, j = ij >> 7;
               const FaceSide& fs = t.side[k & 1];
               const int x = fs.x0 + fs.xi * i + fs.xj * j, y = fs.y0 + fs.yi * i + fs.yj * j, z = fs.z0 + fs.zi * i + fs.zj * j;
               r  = size_t( fs.cell ) * lv.stride + sidx( W, x, y, z );
               si = t.base + faceIndex( N, i, j ) - t.first;
               if ( ( k & 1 ) == 0 )
                  bi = rhs[r];
               partialRow< T, 0, kRowAll >( op, L2Ptr< T >{ u + size_t( fs.cell ) * lv.stride }, fs.cell, W, x, y, z, diag, off );
            }
            diag = groupSum( diag, 2 );
            off  = groupSum( off, 2 );
            bi   = groupSum( bi, 2 );
            const T v = valid ? ( T( 1 ) - relax ) * su[si] + relax * ( bi - off ) / diag : T( 0 );
            __syncwarp(); // both lanes have read su
            if ( valid )
            {
               u[r] = v;
               if ( ( k & 1 ) == 0 )
                  su[si] = v;
            }
         }
      }
      for ( int n = 0; n < nT; ++n )
      {
         const TileDev< T >& t   = tiles[n];
         const int           a   = cnt[0][n][c + 1], e = listEnd( 0, n, c );
         const T             inv = relax / t.diag;
         const int           me  = ( tid + kSurfaceThreads - shift ) % kSurfaceThreads;
         shift                   = ( shift + ( e - a + 31 ) / 32 * 32 ) % kSurfaceThreads;
         for ( int k = a + me; k < e; k += kSurfaceThreads )
         {
            const int ij = deep[k], i = ij & 127, j = ij >> 7;
            const int si = t.base + faceIndex( N, i, j ) - t.first;
            // rows j + 1 and j - 1 hold one point less and one more
            const int up = si + ( N - 1 - j ), dn = si - ( N - j );
            T         off = t.wIn[0] * su[si + 1];
            off += t.wIn[1] * su[si - 1];
            off += t.wIn[2] * su[up];
            off += t.wIn[3] * su[dn];
            off += t.wIn[4] * su[dn + 1];
            off += t.wIn[5] * su[up - 1];
            const T v = ( T( 1 ) - relax ) * su[si] + inv * ( sc[si] - off );
            su[si]    = v; // no point of a colour reads another's value
            u[slabAt( t.side[0], i, j, kSelf )] = v;
            u[slabAt( t.side[1], i, j, kSelf )] = v;
         }
      }
      if ( step + 1 < sf.m )
         grid.sync();
   }
}

size_t surfaceSmem( const SurfaceDev& sf, int elem ) { return size_t( sf.most ) * ( 2 * elem + 2 ) + 16; }

namespace {
// the opt-in to the launch's shared memory in T is set, and the SMs of the current device have room
// for its blocks (a value type whose tiles do not fit is refused by surfaceSor)
template < typename T >
bool prepareFor( const SurfaceDev& sf, int sms )
{
   if ( cudaFuncSetAttribute( k_surface_sor< T >, cudaFuncAttributeMaxDynamicSharedMemorySize, int( kSurfaceMaxSmem ) ) !=
        cudaSuccess )
      return false;
   if ( surfaceSmem( sf, sizeof( T ) ) > kSurfaceMaxSmem )
      return true;
   int perSM = 0;
   return cudaOccupancyMaxActiveBlocksPerMultiprocessor( &perSM, k_surface_sor< T >, kSurfaceThreads,
                                                         surfaceSmem( sf, sizeof( T ) ) ) == cudaSuccess &&
          perSM * sms >= sf.nBlocks;
}

// SMs of the context (or its partition) that the stream's kernels run on; 0 where the driver
// does not say
int streamSMs( cudaStream_t stream )
{
   struct Driver
   {
      CUresult ( *streamCtx )( CUstream, CUcontext*, CUgreenCtx* )                      = nullptr;
      CUresult ( *ctxResource )( CUcontext, CUdevResource*, CUdevResourceType )         = nullptr;
      CUresult ( *greenCtxResource )( CUgreenCtx, CUdevResource*, CUdevResourceType ) = nullptr;
   };
   static const Driver d = [] {
      Driver r;
      auto   get = []( const char* name, auto& f ) {
         void*                           p = nullptr;
         cudaDriverEntryPointQueryResult q;
         if ( cudaGetDriverEntryPointByVersion( name, &p, 12050, cudaEnableDefault, &q ) == cudaSuccess &&
              q == cudaDriverEntryPointSuccess )
            f = reinterpret_cast< std::decay_t< decltype( f ) > >( p );
         else
            cudaGetLastError();
      };
      get( "cuStreamGetCtx", r.streamCtx ); // from 12.5 on: with the stream's green context
      get( "cuCtxGetDevResource", r.ctxResource );
      get( "cuGreenCtxGetDevResource", r.greenCtxResource );
      return r;
   }();
   CUcontext     ctx   = nullptr;
   CUgreenCtx    green = nullptr;
   CUdevResource sm{};
   if ( !d.streamCtx || !d.ctxResource || !d.greenCtxResource || d.streamCtx( stream, &ctx, &green ) != CUDA_SUCCESS )
      return 0;
   const CUresult r = green ? d.greenCtxResource( green, &sm, CU_DEV_RESOURCE_TYPE_SM )
                            : d.ctxResource( ctx, &sm, CU_DEV_RESOURCE_TYPE_SM );
   return r == CUDA_SUCCESS ? int( sm.sm.smCount ) : 0;
}
} // namespace

bool surfacePrepare( const SurfaceDev& sf )
{
   int        dev = 0, coop = 0, mps = 0, sms = 0;
   const bool ok  = cudaGetDevice( &dev ) == cudaSuccess &&
                   cudaDeviceGetAttribute( &coop, cudaDevAttrCooperativeLaunch, dev ) == cudaSuccess && coop &&
                   cudaDeviceGetAttribute( &mps, cudaDevAttrMpsEnabled, dev ) == cudaSuccess && !mps &&
                   cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev ) == cudaSuccess &&
                   prepareFor< float >( sf, sms ) && prepareFor< double >( sf, sms );
   if ( !ok )
      cudaGetLastError(); // a query the device or driver refuses is an answer, not an error of the storage
   return ok;
}

template < typename T >
cudaError_t launchSurfaceSor( const TopoDev& tp, const LevelDev& lv, const SurfaceDev& sf, const OpDev< T >& op, T* u,
                              const T* rhs, T relax, bool backwards, cudaStream_t stream )
{
   // A captured launch is refused only when its graph is instantiated or run, so the grid is
   // held against the stream's SMs here (one resident block each) and not left to the launch.
   if ( streamSMs( stream ) < sf.nBlocks )
      return cudaErrorCooperativeLaunchTooLarge;
   cudaLaunchConfig_t  c{};
   cudaLaunchAttribute a{};
   a.id               = cudaLaunchAttributeCooperative;
   a.val.cooperative  = 1;
   c.gridDim          = dim3( unsigned( sf.nBlocks ) );
   c.blockDim         = dim3( kSurfaceThreads );
   c.dynamicSmemBytes = surfaceSmem( sf, sizeof( T ) );
   c.stream           = stream;
   c.attrs            = &a;
   c.numAttrs         = 1;
   return cudaLaunchKernelEx( &c, k_surface_sor< T >, tp, lv, sf, op, u, rhs, relax, backwards ? 1 : 0 );
}

template cudaError_t launchSurfaceSor< float >( const TopoDev&, const LevelDev&, const SurfaceDev&, const OpDev< float >&,
                                                float*, const float*, float, bool, cudaStream_t );
template cudaError_t launchSurfaceSor< double >( const TopoDev&, const LevelDev&, const SurfaceDev&, const OpDev< double >&,
                                                 double*, const double*, double, bool, cudaStream_t );

} // namespace hyb
