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

SurfaceDev tiles()
{
   SurfaceDev sf{};
   sf.nBlocks = 148;
   sf.most    = 8000; // 144 KB in FP64
   return sf;
}

// two devices of one process, each with its own storage: both launch above 48 KB
int devices()
{
   const SurfaceDev sf = tiles();
   for ( fake.device = 0; fake.device < 2; ++fake.device )
   {
      CHECK( surfacePrepare( sf ) );
      CHECK( launch< double >( sf ) == cudaSuccess );
      CHECK( launch< float >( sf ) == cudaSuccess );
   }
   CHECK( fake.launches == 4 );
   return 0;
}

// whether a storage keeps its tiles: decided when it is built, so that no solve that is captured
// into a graph holds a launch the device cannot run
int fits()
{
   auto kept = []( auto&& change ) {
      fake = FakeCuda{};
      change();
      return surfacePrepare( tiles() );
   };
   CHECK( kept( [] {} ) );
   CHECK( !kept( [] { fake.mps = 1; } ) );
   CHECK( !kept( [] { fake.cooperative = 0; } ) );
   CHECK( !kept( [] { fake.perSM = 0; } ) );
   CHECK( !kept( [] { fake.refuses = true; } ) ); // and the storage is built all the same
   CHECK( !kept( [] { fake.sms = 147; } ) );
   CHECK( kept( [] { fake.sms = 74, fake.perSM = 2; } ) );
   return 0;
}

// a stream on a part of the device: refused before anything is launched or captured
int stream()
{
   const SurfaceDev sf = tiles();
   auto             launched = [&]( auto&& change ) {
      fake = FakeCuda{};
      change();
      return surfacePrepare( sf ) && launch< float >( sf ) == cudaSuccess && fake.launches == 1;
   };
   CHECK( launched( [] {} ) );
   CHECK( !launched( [] { fake.greenSMs = 64; } ) );
   CHECK( launch< float >( sf ) == cudaErrorCooperativeLaunchTooLarge && fake.launches == 0 );
   CHECK( launched( [] { fake.greenSMs = 148; } ) );
   CHECK( !launched( [] { fake.ctxSMs = 100; } ) );
   return 0;
}

// a driver that does not say how many SMs a stream has
int silent()
{
   fake.noDriver = true;
   CHECK( surfacePrepare( tiles() ) );
   CHECK( launch< double >( tiles() ) == cudaErrorCooperativeLaunchTooLarge && fake.launches == 0 );
   return 0;
}

int main( int, char** argv )
{
   struct
   {
      const char* name;
      int ( *f )();
   } const checks[] = { { "devices", devices }, { "fits", fits }, { "stream", stream }, { "silent", silent } };
   for ( const auto& c : checks )
      if ( !std::strcmp( argv[1], c.name ) )
         return c.f();
   return 2;
}
