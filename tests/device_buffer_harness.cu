// Host-side checks of the library's device buffers on the stand-in runtime
// (fake_cudart.cpp).
#include "cipc_internal.h"

extern "C" void fake_fail_malloc(int nth);

// 1 where a buffer whose growth failed is whole again after a smaller request,
// and a launch after that would not be taken for failed
extern "C" int buffer_recovers(int first, int failing, int again) {
    cipc::DBuf<double> d;
    d.reserve(first);
    fake_fail_malloc(1);
    bool failed = false;
    try {
        d.reserve(failing);
    } catch (const cipc::CudaError&) {
        failed = true;
    }
    fake_fail_malloc(0);
    d.reserve(again);
    const bool whole = failed && d.p && d.cap >= (size_t)again && cudaPeekAtLastError() == cudaSuccess;
    d.free();
    return whole;
}
