// The CUDA runtime functions that hyb_surface.cu and its check use, on devices that exist only
// here: a kernel's shared-memory opt-in is kept per device, as the runtime keeps it.
#include "fake_cudart.hpp"

#include <cstring>
#include <map>

#include <cuda.h>

FakeCuda fake;

namespace {
std::map< const void*, int > optIn[2]; // by device: kernel -> bytes of dynamic shared memory allowed
int                          a_green;

CUresult streamCtx( CUstream, CUcontext* c, CUgreenCtx* g )
{
   *c = nullptr;
   *g = fake.greenSMs ? reinterpret_cast< CUgreenCtx >( &a_green ) : nullptr;
   return CUDA_SUCCESS;
}
CUresult ctxResource( CUcontext, CUdevResource* r, CUdevResourceType )
{
   r->sm.smCount = unsigned( fake.ctxSMs );
   return CUDA_SUCCESS;
}
CUresult greenResource( CUgreenCtx, CUdevResource* r, CUdevResourceType )
{
   r->sm.smCount = unsigned( fake.greenSMs );
   return CUDA_SUCCESS;
}
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
cudaError_t cudaGetDevice( int* d )
{
   *d = fake.device;
   return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute( int* v, cudaDeviceAttr a, int )
{
   if ( fake.refuses )
      return cudaErrorInvalidValue;
   *v = a == cudaDevAttrCooperativeLaunch ? fake.cooperative : a == cudaDevAttrMpsEnabled ? fake.mps : fake.sms;
   return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags( int* n, const void*, int, size_t, unsigned )
{
   *n = fake.perSM;
   return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor( int* n, const void*, int, size_t )
{
   *n = fake.perSM;
   return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion( const char* name, void** f, unsigned, unsigned long long,
                                              cudaDriverEntryPointQueryResult* q )
{
   *f = !std::strcmp( name, "cuStreamGetCtx" )        ? reinterpret_cast< void* >( streamCtx )
        : !std::strcmp( name, "cuCtxGetDevResource" ) ? reinterpret_cast< void* >( ctxResource )
                                                      : reinterpret_cast< void* >( greenResource );
   *q = fake.noDriver ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
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
