// Host-side internals of libpff: status/error plumbing and workspace carving.
#pragma once
#include <cstddef>
#include <cstdint>
#include <atomic>
#include <cstdio>
#include <cuda_runtime.h>
#include "../../include/pff.h"
#include "pff_common.cuh"

namespace pff {

// Number of kernels this library has launched (all threads); read by benchmarks.
extern std::atomic<long long> g_launches;
inline void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

// Timing probes (pff_probe_enable / pff_probe_read): PFF_PROBED(name, stream, launch)
// brackets `launch` with events on `stream` while probes are armed.
struct ProbeMark {
    int slot, idx;
};
ProbeMark probe_begin(const char *name, cudaStream_t st);
void probe_end(ProbeMark m, cudaStream_t st);
#define PFF_PROBED(name, st, ...)                                 \
    do {                                                          \
        const ::pff::ProbeMark _pm = ::pff::probe_begin(name, st); \
        __VA_ARGS__;                                              \
        ::pff::probe_end(_pm, st);                                \
    } while (0)

void set_error(const char *fmt, ...);
void clear_error();

// Internal status (never returned through the C ABI): a fast path that is not
// available here, so the caller takes its general path.
constexpr int PFF_ERR_UNSUPPORTED = 100;

// Returns PFF_ERR_CUDA (and records where) if the last launch/copy failed.
int check_cuda(const char *where);

#define PFF_TRY(expr)                         \
    do {                                      \
        int _rc = (expr);                     \
        if (_rc != PFF_OK) return _rc;        \
    } while (0)

#define PFF_CUDA(call)                                                     \
    do {                                                                   \
        cudaError_t _e = (call);                                           \
        if (_e != cudaSuccess) {                                           \
            ::pff::set_error("%s: %s", #call, cudaGetErrorString(_e));    \
            return PFF_ERR_CUDA;                                           \
        }                                                                  \
    } while (0)

int check_grid(int nx, int ny, int mode, const uint8_t *codes);

// Read small device int arrays (a list of (pointer, count), at most 8 pointers and
// 64 ints) into host memory, in order, and synchronise `st`.  A one-thread kernel
// stores them into mapped pinned host memory, so the read uses no copy engine and
// does not wait behind bulk transfers other streams have in flight.
struct IntReads {
    const int *src[8];
    int n[8];
    int k = 0;
    IntReads &add(const int *p, int cnt)
    {
        src[k] = p;
        n[k++] = cnt;
        return *this;
    }
};
int read_ints(const IntReads &r, int *out, cudaStream_t st);

// The calling thread's 64 pinned ints on the current device: host and device address.
int pinned_ints(int **host, int **dptr);


// Bump allocator over a caller-provided device workspace (256-byte aligned slices).
struct Carver {
    char *base;
    size_t cap, off;
    Carver(void *b, size_t c) : base((char *)b), cap(c), off(0) {}
    template <class T>
    T *take(size_t n)
    {
        size_t a = (off + 255) & ~size_t(255);
        off = a + n * sizeof(T);
        return (off <= cap && base) ? (T *)(base + a) : nullptr;
    }
    static size_t round(size_t n) { return (n + 255) & ~size_t(255); }
};

// How long the blocks of a cooperative launch wait at a barrier, and for how many more blocks
// than there are (pff_barrier_test; otherwise two seconds and none).
enum { BAR_REROUTE = 1, BAR_LABELS = 2, BAR_TREE = 4, BAR_ROUNDS = 8 };
struct BarWait {
    int absent;
    unsigned limit_us;
};
BarWait bar_wait(int kernel);

// A tile of a ragged batch.
struct BatchTile {
    long long off;   // first cell of the tile in the packed arrays
    long long boff;  // first basin entry (N+1 entries per tile)
    int nx, ny, mode;
    int id;          // the tile's index in the caller's order
    float dx;
    int item0;       // its first work item of the accumulation front, -1: accumulated by its own CTA
    int logn;        // rake-and-compress rounds: ceil(log2 N) + 1
    int pad;
};

// error bits of a batch's status word
enum : int { BST_MODE = 1, BST_CYCLE_LABELS = 8, BST_CARVE = 16, BST_ROUNDS = 32 };

// The accumulation of a ragged batch (pff_accum.cu), over packed arrays.
constexpr int BATCH_ACC_CTR = 256;
struct BatchAcc {
    const int32_t *rcv;
    float *Q;             // in: seeds, out: sums
    uint32_t *counts;
    void *bufA, *bufB, *priv;  // 16 B per cell each
    int *la[2], *lf[2];   // 4 B per cell each
    int *ctr;             // BATCH_ACC_CTR ints, zero
    const int *small;     // null, or whether the sums are there already
    int *status;          // BST_* bits
    const BatchTile *by_offset;  // the tiles in packed order
    const int *items;     // work item -> tile (packed order)
    const int *limits;    // [0] smallest and [1] largest logn of the front's tiles, [2] work items
    long long total;
    int ntiles;
};
bool batch_front_takes(int nx, int ny, int mode);
int batch_front_items(int nx, int ny);
int launch_batch_accumulate(const BatchAcc &b, cudaStream_t st);

inline cudaStream_t S(void *s) { return (cudaStream_t)s; }

// Launch helpers implemented per translation unit (declared for cross-TU use).
int launch_basin_init(int32_t *bid, const Grid &g, cudaStream_t st);
int run_labels(int32_t *bid, int32_t *rec_work, const Grid &g, int *round_flags, cudaStream_t st);
int count_pits(const int32_t *rec, const Grid &g, int *dev_count, int *pit_list, int *host_count,
               cudaStream_t st);

}  // namespace pff
