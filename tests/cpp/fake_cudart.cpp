// The CUDA runtime functions that hyb_surface.cu and its check use, on devices that exist only
// here: a kernel's shared-memory opt-in is kept per device, as the runtime keeps it.
#include "fake_cudart.hpp"

#include <map>

FakeCuda fake;

namespace {
std::map< const void*, int > optIn[2]; // by device: kernel -> bytes of dynamic shared memory allowed
}

extern "C" {

char   __cudaInitModule( void** ) { return 1; }
void** __cudaRegisterFatBinary( void* )
{
   static void* h;
   return &h;
}
void __cudaRegisterFatBinaryEnd( void** ) {}
void __cudaUnregisterFatBinary( void** ) {}
void __cudaRegisterFunction( void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int* ) {}
void __cudaRegisterVar( void**, char*, char*, const char*, int, size_t, int, int ) {}
unsigned    __cudaPushCallConfiguration( dim3, dim3, size_t, void* ) { return 0; }
cudaError_t __cudaPopCallConfiguration( dim3*, dim3*, size_t*, void* ) { return cudaSuccess; }
cudaError_t cudaLaunchKernel( const void*, dim3, dim3, void**, size_t, cudaStream_t ) { return cudaErrorNotSupported; }

cudaError_t cudaFuncSetAttribute( const void* f, cudaFuncAttribute a, int v )
{
   if ( a == cudaFuncAttributeMaxDynamicSharedMemorySize )
      optIn[fake.device][f] = v;
   return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC( const cudaLaunchConfig_t* c, const void* f, void** )
{
   const auto it = optIn[fake.device].find( f );
   if ( c->dynamicSmemBytes > size_t( it == optIn[fake.device].end() ? 48 * 1024 : it->second ) )
      return cudaErrorInvalidValue;
   ++fake.launches;
   return cudaSuccess;
}
}
