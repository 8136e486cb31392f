// Internal: context object behind the opaque lcc_ctx of include/livecc_b200.h.
#pragma once
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

struct lcc_ctx {
    int device;
    int num_sms;
    int* fault;      // mapped host memory, written by kernels only: a bounded wait inside a product gave up. Stays set
    char err[512];
};

#define LCC_FAIL(ctx, code, ...)                               \
    do {                                                       \
        if (ctx) snprintf((ctx)->err, sizeof((ctx)->err), __VA_ARGS__); \
        return (code);                                         \
    } while (0)

// A fault that a kernel of an earlier call recorded is found by the next call, or by lcc_check_fault() once the stream is synchronised.
#define LCC_CHECK_FAULT(ctx, what)                                                         \
    do {                                                                                   \
        if ((ctx)->fault && *(volatile int*)(ctx)->fault)                                  \
            LCC_FAIL(ctx, -101, "%s: a bounded wait inside a matrix product gave up; results of this context are invalid from there on", what); \
    } while (0)

#define LCC_CHECK_LAUNCH(ctx, what)                                                        \
    do {                                                                                   \
        LCC_CHECK_FAULT(ctx, what);                                                        \
        cudaError_t e__ = cudaGetLastError();                                              \
        if (e__ != cudaSuccess) LCC_FAIL(ctx, -100, "%s: %s", what, cudaGetErrorString(e__)); \
    } while (0)
