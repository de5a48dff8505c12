/* A communicator whose ranks are threads of one process on one GPU, with NCCL's names (libnccl.so.2 to the library under
 * test): what the ranks exchange goes through host memory, and nothing on the GPU waits for another rank.  Every wait
 * here ends after 30 s with an error. */
#include <cuda_runtime.h>
#include <nccl.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <string.h>
#include <time.h>

enum { kRanks = 8, kBytes = 64 * 1024 };
struct ncclComm {
    int rank;
};
static atomic_int arrived, generation;
static int n_ranks;
static char box[kRanks][kBytes];

static ncclResult_t meet(int ranks) {
    const int mine = atomic_load(&generation);
    if (atomic_fetch_add(&arrived, 1) + 1 == ranks) {
        atomic_store(&arrived, 0);
        atomic_fetch_add(&generation, 1);
        return ncclSuccess;
    }
    const time_t t0 = time(NULL);
    while (atomic_load(&generation) == mine)
        if (time(NULL) - t0 > 30) return ncclSystemError;
    return ncclSuccess;
}

ncclResult_t ncclGetUniqueId(ncclUniqueId* id) {
    struct timespec t;
    clock_gettime(CLOCK_REALTIME, &t);
    memset(id, 0, sizeof *id);
    memcpy(id, &t, sizeof t);
    return ncclSuccess;
}
ncclResult_t ncclCommInitRank(ncclComm_t* comm, int ranks, ncclUniqueId id, int rank) {
    (void)id;
    if (ranks > kRanks || !(*comm = malloc(sizeof **comm))) return ncclSystemError;
    (*comm)->rank = rank;
    n_ranks = ranks;
    return meet(ranks);
}
ncclResult_t ncclCommDestroy(ncclComm_t comm) {
    free(comm);
    return ncclSuccess;
}
ncclResult_t ncclCommAbort(ncclComm_t comm) { return ncclCommDestroy(comm); }
ncclResult_t ncclAllGather(const void* send, void* recv, size_t count, ncclDataType_t type, ncclComm_t comm, cudaStream_t stream) {
    if (type != ncclUint8 || count > kBytes) return ncclInvalidArgument;
    if (cudaMemcpyAsync(box[comm->rank], send, count, cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
        return ncclSystemError;
    ncclResult_t r = meet(n_ranks);
    if (r != ncclSuccess) return r;
    for (int q = 0; q < n_ranks; q++)
        if (cudaMemcpyAsync((char*)recv + q * count, box[q], count, cudaMemcpyHostToDevice, stream) != cudaSuccess) return ncclSystemError;
    if (cudaStreamSynchronize(stream) != cudaSuccess) return ncclSystemError;
    return meet(n_ranks);
}
const char* ncclGetErrorString(ncclResult_t r) { return r == ncclSuccess ? "success" : "error"; }
ncclResult_t ncclCommGetAsyncError(ncclComm_t comm, ncclResult_t* r) {
    (void)comm;
    *r = ncclSuccess;
    return ncclSuccess;
}
