#pragma once
#include <cuda_runtime_api.h>

struct FakeCuda
{
   int device      = 0; // the current one
   int launches    = 0;
   int sms         = 148; // of the device
   int cooperative = 1;   // the device can run cooperative launches
   int mps         = 0;   // its contexts are shared via MPS
   int perSM       = 1;   // resident blocks of any kernel per SM
   int ctxSMs      = 148; // of a stream's context
   int greenSMs    = 0;   // of a stream's green context (0: it has none)
   bool refuses    = false; // attribute queries fail
   bool noDriver   = false; // the driver's entry points are not found
};
extern FakeCuda fake;
