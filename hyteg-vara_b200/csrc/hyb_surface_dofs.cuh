// Micro-vertices on macro-vertices, -edges and -faces: their enumeration, their rows summed
// over the adjacent cells, and the writes to all their replicas.
#pragma once

#include "hyb_device.cuh"

namespace hyb {

// ---------------------------------------------------------------------------
// Boundary-DoF enumeration: [vertices | edge interiors | face interiors]
// ---------------------------------------------------------------------------
struct BdryPoint
{
   int kind, prim, i, j;
};

__device__ __forceinline__ BdryPoint decodeBdry( const TopoDev& tp, const LevelDev& lv, int t )
{
   BdryPoint p{ 0, 0, 0, 0 };
   if ( t < tp.nV )
   {
      p.kind = 0;
      p.prim = t;
      return p;
   }
   t -= tp.nV;
   const int ne = tp.nE * ( lv.N - 1 );
   if ( t < ne )
   {
      p.kind = 1;
      p.prim = t / ( lv.N - 1 );
      p.i    = t % ( lv.N - 1 ) + 1;
      return p;
   }
   t -= ne;
   p.kind = 2;
   p.prim = t / lv.nIntFace;
   const int q  = t % lv.nIntFace;
   const int rr = lv.nIntFace - 1 - q; // index counted from the short rows
   int       k  = int( ( sqrtf( 8.0f * float( rr ) + 1.0f ) - 1.0f ) * 0.5f );
   while ( ( k + 1 ) * ( k + 2 ) / 2 <= rr )
      ++k;
   while ( k * ( k + 1 ) / 2 > rr )
      --k;
   p.i = ( k + 1 ) * ( k + 2 ) / 2 - 1 - rr + 1;
   p.j = lv.N - 2 - k;
   return p;
}

__device__ __forceinline__ int numEmb( const TopoDev& tp, int kind, int prim )
{
   if ( kind == 2 )
      return tp.fEmb[2 * prim + 1] >= 0 ? 2 : 1;
   if ( kind == 1 )
      return tp.eEmbOff[prim + 1] - tp.eEmbOff[prim];
   return tp.vEmbOff[prim + 1] - tp.vEmbOff[prim];
}
__device__ __forceinline__ int32_t embAt( const TopoDev& tp, int kind, int prim, int e )
{
   if ( kind == 2 )
      return tp.fEmb[2 * prim + e];
   if ( kind == 1 )
      return tp.eEmb[tp.eEmbOff[prim] + e];
   return tp.vEmb[tp.vEmbOff[prim] + e];
}
__device__ __forceinline__ uint8_t primBc( const TopoDev& tp, int kind, int prim )
{
   return kind == 2 ? tp.fBc[prim] : kind == 1 ? tp.eBc[prim] : tp.vBc[prim];
}

// Full row (sum of partial rows over adjacent cells) of a boundary DoF.
template < typename T, int VAR >
__device__ __forceinline__ void bdryRow( const TopoDev& tp, const LevelDev& lv, const OpDev< T >& op, const T* u,
                                         const BdryPoint& p, T& diag, T& off )
{
   const int ne = numEmb( tp, p.kind, p.prim );
   for ( int e = 0; e < ne; ++e )
   {
      int c, x, y, z;
      embeddingCoords( embAt( tp, p.kind, p.prim, e ), p.kind, lv.N, p.i, p.j, c, x, y, z );
      partialRow< T, VAR >( op, u + size_t( c ) * lv.stride, c, lv.W, x, y, z, diag, off );
   }
}

template < typename T >
__device__ __forceinline__ size_t bdryReplica( const TopoDev& tp, const LevelDev& lv, const BdryPoint& p, int e )
{
   int c, x, y, z;
   embeddingCoords( embAt( tp, p.kind, p.prim, e ), p.kind, lv.N, p.i, p.j, c, x, y, z );
   return size_t( c ) * lv.stride + sidx( lv.W, x, y, z );
}

template < typename T >
__device__ __forceinline__ void bdryWriteAll( const TopoDev& tp, const LevelDev& lv, const BdryPoint& p, T* dst, T v )
{
   const int ne = numEmb( tp, p.kind, p.prim );
   for ( int e = 0; e < ne; ++e )
      dst[bdryReplica< T >( tp, lv, p, e )] = v;
}

// ---------------------------------------------------------------------------
// Lane groups for surface DoFs. A DoF on a macro-vertex gets 32 lanes, on a
// macro-edge 8, on a macro-face 2; lane `sub` of the group handles the adjacent
// cells e = sub, sub + G, ... and the group reduces with warp shuffles. Each kind's
// lane range is padded to whole warps, so all lanes of a warp share G and every
// shuffle is executed by the full warp.
// ---------------------------------------------------------------------------
struct BdryLists
{
   const int32_t* v; // surface-DoF indices of each kind, or nullptr for the full range
   const int32_t* e;
   const int32_t* f;
   int            nv, ne, nf;
};

__device__ __forceinline__ BdryLists fullBdryLists( const TopoDev& tp, const LevelDev& lv )
{
   return BdryLists{ nullptr, nullptr, nullptr, tp.nV, tp.nE * ( lv.N - 1 ), tp.nF * lv.nIntFace };
}

__host__ __device__ __forceinline__ long bdryLaneCount( int nv, int ne, int nf )
{
   return long( nv ) * 32 + ( long( ne ) * 8 + 31 ) / 32 * 32 + ( long( nf ) * 2 + 31 ) / 32 * 32;
}

struct LaneTask
{
   int  t;      // surface-DoF index in [vertices | edge interiors | face interiors]
   int  G, sub; // group size and lane within the group
   bool valid;  // false for padding lanes
};

__device__ __forceinline__ LaneTask laneTask( const TopoDev& tp, const LevelDev& lv, const BdryLists& bl, long gt )
{
   LaneTask  tk{ 0, 32, 0, false };
   const long nvl = long( bl.nv ) * 32, nel = ( long( bl.ne ) * 8 + 31 ) / 32 * 32;
   if ( gt < nvl )
   {
      const int idx = int( gt >> 5 );
      tk            = { bl.v ? bl.v[idx] : idx, 32, int( gt & 31 ), true };
   }
   else if ( ( gt -= nvl ) < nel )
   {
      const int idx = int( gt >> 3 );
      tk.G          = 8;
      tk.sub        = int( gt & 7 );
      tk.valid      = idx < bl.ne;
      tk.t          = tk.valid ? ( bl.e ? bl.e[idx] : tp.nV + idx ) : 0;
   }
   else
   {
      gt -= nel;
      const int idx = int( gt >> 1 );
      tk.G          = 2;
      tk.sub        = int( gt & 1 );
      tk.valid      = idx < bl.nf;
      tk.t          = tk.valid ? ( bl.f ? bl.f[idx] : tp.nV + tp.nE * ( lv.N - 1 ) + idx ) : 0;
   }
   return tk;
}

template < typename T >
__device__ __forceinline__ T groupSum( T v, int G )
{
   for ( int o = G >> 1; o > 0; o >>= 1 )
      v += __shfl_xor_sync( 0xffffffffu, v, o );
   return v;
}

// Partial rows of the group's adjacent cells, summed over the group (all lanes get it).
template < typename T, int VAR, int LOADS = rowLoads< T >() >
__device__ __forceinline__ void bdryRowGroup( const TopoDev& tp, const LevelDev& lv, const OpDev< T >& op, const T* u,
                                              const BdryPoint& p, const LaneTask& tk, bool active, T& diag, T& off )
{
   diag = 0;
   off  = 0;
   if ( active )
   {
      const int ne = numEmb( tp, p.kind, p.prim );
      for ( int e = tk.sub; e < ne; e += tk.G )
      {
         int c, x, y, z;
         embeddingCoords( embAt( tp, p.kind, p.prim, e ), p.kind, lv.N, p.i, p.j, c, x, y, z );
         partialRow< T, VAR, LOADS >( op, u + size_t( c ) * lv.stride, c, lv.W, x, y, z, diag, off );
      }
   }
   diag = groupSum( diag, tk.G );
   off  = groupSum( off, tk.G );
}

template < typename T >
__device__ __forceinline__ void bdryWriteGroup( const TopoDev& tp, const LevelDev& lv, const BdryPoint& p,
                                                const LaneTask& tk, T* dst, T v )
{
   const int ne = numEmb( tp, p.kind, p.prim );
   for ( int e = tk.sub; e < ne; e += tk.G )
      dst[bdryReplica< T >( tp, lv, p, e )] = v;
}

} // namespace hyb
