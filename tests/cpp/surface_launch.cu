// Host side of the one-launch interface passes (hyb_surface.cu) against a fake CUDA runtime.
#include "fake_cudart.hpp"
#include "hyb_surface.hpp"

#include <cstdio>
#include <cstring>

using namespace hyb;

#define CHECK( c )                                                   \
   do                                                                \
      if ( !( c ) )                                                  \
      {                                                              \
         std::printf( "line %d: %s\n", __LINE__, #c );               \
         return 1;                                                   \
      }                                                              \
   while ( 0 )

template < typename T >
cudaError_t launch( const SurfaceDev& sf )
{
   TopoDev    tp{};
   LevelDev   lv{};
   OpDev< T > op{};
   return launchSurfaceSor< T >( tp, lv, sf, op, nullptr, nullptr, T( 1 ), false, nullptr );
}

// two devices of one process, each with its own storage: both launch above 48 KB
int devices()
{
   SurfaceDev sf{};
   sf.nBlocks = 148;
   sf.most    = 8000; // 144 KB in FP64
   for ( fake.device = 0; fake.device < 2; ++fake.device )
   {
      CHECK( surfacePrepare() == cudaSuccess );
      CHECK( launch< double >( sf ) == cudaSuccess );
      CHECK( launch< float >( sf ) == cudaSuccess );
   }
   CHECK( fake.launches == 4 );
   return 0;
}

int main( int, char** argv )
{
   if ( !std::strcmp( argv[1], "devices" ) )
      return devices();
   return 2;
}
