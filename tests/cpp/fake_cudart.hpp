#pragma once
#include <cuda_runtime_api.h>

struct FakeCuda
{
   int device   = 0; // the current one
   int launches = 0;
};
extern FakeCuda fake;
