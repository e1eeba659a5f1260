/* A solver's rate tables: device memory for the temperature part of the rates
 * of a solve's cells, [cells][reactions], filled by every solve that uses it.
 *
 * A table is optional (without one the solve kernel evaluates the rates, with
 * the same results), so it gives way to everything else: it is taken only
 * where it leaves half of the free memory, and drop() gives it back
 * for buffers that a solve cannot do without.  A larger table replaces the
 * one before it.  Only a table used under stream capture stays until close(),
 * since the graph holds its address; the next one then is at least twice as
 * large, so that such tables together take less than the newest does.
 *
 * Plain runtime calls only, so that this file compiles without a device
 * compiler. */
#ifndef OV_RATE_TABLES_HPP
#define OV_RATE_TABLES_HPP

#include <cuda_runtime_api.h>
#include <stddef.h>
#include <stdint.h>

namespace ov {

/* Another thread or stream may be capturing in the default (global) mode, in
   which an allocation anywhere fails and spoils the capture; the allocations
   here belong to no graph */
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

struct RateTables {
    static constexpr int MAX = 48; /* doubling sizes: never reached */
    int n;
    bool captured; /* the newest table is in a graph, as all before it are */
    int64_t cells[MAX];
    double* tab[MAX];

    /* a table of at least ncells cells of nrea doubles for a solve on st, or
       null: no room, or a capture that would have to allocate it */
    double* get(int64_t ncells, int64_t nrea, cudaStream_t st)
    {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        bool capturing = true; /* also the legacy stream beside a capture */
        if (cudaStreamIsCapturing(st, &cap) == cudaSuccess)
            capturing = cap != cudaStreamCaptureStatusNone;
        else
            cudaGetLastError();
        if (n == 0 || cells[n - 1] < ncells) {
            if (capturing)
                return nullptr;
            /* the first of the size asked for, later ones with some room */
            int64_t want = n > 0 ? ncells + ncells / 8 : ncells;
            drop();
            if (n > 0 && want < 2 * cells[n - 1])
                want = 2 * cells[n - 1];
            if (n == MAX)
                return nullptr;
            const size_t bytes = sizeof(double) * (size_t)nrea * (size_t)want;
            RelaxedCapture relaxed;
            size_t room = 0, total = 0;
            void* p = nullptr;
            if (cudaMemGetInfo(&room, &total) != cudaSuccess || bytes > room / 2 ||
                cudaMalloc(&p, bytes) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            tab[n] = (double*)p;
            cells[n++] = want;
            captured = false;
        }
        captured = captured || capturing;
        return tab[n - 1];
    }

    /* gives the newest table back unless a graph may hold it; true if memory
       became free */
    bool drop()
    {
        if (n == 0 || captured)
            return false;
        RelaxedCapture relaxed;
        cudaFree(tab[--n]); /* waits for the kernels that use it */
        captured = n > 0;
        return true;
    }

    /* cudaMalloc for a buffer that a solve cannot do without: where there is no
       room, the newest table gives way */
    template <class T>
    cudaError_t alloc(T** p, size_t bytes)
    {
        cudaError_t e = cudaMalloc((void**)p, bytes);
        if (e == cudaErrorMemoryAllocation && drop())
            e = cudaMalloc((void**)p, bytes);
        if (e != cudaSuccess)
            cudaGetLastError(); /* the caller returns it */
        return e;
    }

    void close()
    {
        while (n > 0)
            cudaFree(tab[--n]);
        captured = false;
    }
};

}  // namespace ov

#endif /* OV_RATE_TABLES_HPP */
