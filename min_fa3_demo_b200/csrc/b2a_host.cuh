// Host-side helpers shared by the C-ABI entry points: error text, device checks,
// tensor-map construction, workspace layout.
#pragma once

#include <algorithm>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/b200attn.h"

namespace b2a {

// Thread-local error text behind b2a_last_error().
char* error_buffer();
int fail(int code, const char* fmt, ...);

#define B2A_CUDA_OK(expr)                                                             \
    do {                                                                              \
        cudaError_t err__ = (expr);                                                   \
        if (err__ != cudaSuccess) {                                                   \
            return ::b2a::fail(B2A_ERR_CUDA, "%s failed: %s", #expr,                  \
                               cudaGetErrorString(err__));                            \
        }                                                                             \
    } while (0)

#define B2A_REQUIRE(cond, ...)                                         \
    do {                                                               \
        if (!(cond)) {                                                 \
            return ::b2a::fail(B2A_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
        }                                                              \
    } while (0)

struct DeviceInfo {
    int device;
    int sm_count;
    int cc_major;
    int cc_minor;
    int max_smem_optin;
};

// Cached per-device properties of the current device (requires compute capability 10.x).
int current_device_info(DeviceInfo* info);

// 3-D tiled tensor map over a flat bf16 [tokens, heads, 128] tensor with a
// (64 columns, box_heads heads, box_rows tokens) box and 128-byte swizzle.
int make_token_map(CUtensorMap* map, const void* base, uint64_t tokens, uint64_t heads,
                   uint32_t box_rows, uint32_t box_heads = 1);

// Header words at the start of every workspace.
struct WorkspaceHeader {
    int sched_counter;        // dynamic tile scheduler ticket; -n: no tickets, and n status words, one for each CTA, behind the header
    int num_entries;          // varlen: number of planned work-list entries
    unsigned int status;      // device status word (0 = ok)
    int reserved;
};
static_assert(sizeof(WorkspaceHeader) == 16, "workspace header is 16 bytes");

// Launches a kernel that begins with wait_for_previous_kernel (after what needs no global memory): its CTAs may come up while
// the stream's previous kernel ends, which takes the launch, barriers, tensor memory and descriptors off the path.  Such a
// kernel lives while that one still writes, so no pointer of it is __restrict__ const and nothing is read through the
// read-only path: both promise that the data does not change while the kernel lives.  Used by the
// forward's kernels and the planner (us, without / with: 1 x 128, 32 heads 10.6 / 9.2; 16,384 tokens in short documents, two
// kernels, 78.6 / 75.7; one token for 16 x 4,001 46.7 / 45.4; 512 rows against 16,384 keys, two kernels, 128.7 / 126.6), not by
// the backward's: its CTAs then start one by one as the preprocess ends and stay out of step (4 x 8,192 causal 4,995 / 5,119;
// 4,096 without a mask 670 / 687).
template <typename... Params, typename... Args>
cudaError_t launch_early(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// Room for such words in a fixed-length forward's workspace (a B200 has 148 SMs; the rest is for copy CTAs): 1 KiB with the header.
constexpr int kFwdStatusWords = 252;

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Upper bound on work-list entries when documents are cut into `rows`-token pieces.
inline size_t max_entries(int batch, int total_tokens, int rows) {
    return static_cast<size_t>(total_tokens) / rows + static_cast<size_t>(batch) + 1;
}

constexpr uint32_t kDefaultTimeoutNs = 2000000000u;   // bounded device waits: 2 s
constexpr uint32_t kMaxTimeoutNs = 4000000000u;       // the waits compare 32-bit nanosecond timers

// Limit of every bounded device-side wait of launches made from now on (b2a_set_wait_timeout_ns).
uint32_t wait_timeout_ns();
// Limit of the cross-rank completion wait that ends the context-parallel backward: ten times
// the limit above, because it covers the other ranks' whole backward launch and their launch skew.
unsigned long long completion_timeout_ns();

// Device address of the scratch array built into the library for b2a_fwd_noalloc (looked up
// once per device with cudaGetSymbolAddress; defined beside the array in b2a_fwd.cu).
int noalloc_scratch_ptr(void** out);

// Runs `fn` once per (device, slot) under a lock; used for cudaFuncSetAttribute calls.
// Returns fn's code the first time and B2A_OK afterwards.
int once_per_device(int device, int slot, int (*fn)());

// How long a list of work items takes when each CTA takes the next item as soon as it is done with its last, in the unit of
// the items' lengths (whole steps).  Times are kept as counts of CTAs per step, so an add() of equal items costs a few
// instructions and the whole a microsecond or two.
class HandOut {
public:
    // total, longest: at least the sum and the maximum of all lengths that will be added (they set the resolution).
    HandOut(int ctas, double total, double longest) : unit_(1 + static_cast<int>((total / ctas + longest) / (kSlots / 2))) {
        // Nothing starts later than the mean load, so times end at total / ctas + longest; half the room is spare.
        slots_ = std::min(kSlots, 64 + 2 * static_cast<int>((total / ctas + longest) / unit_));
        std::fill(free_, free_ + slots_, 0);
        free_[0] = ctas;
    }
    void add(int length, long long times) {
        const int d = (length + unit_ - 1) / unit_;
        while (times > 0) {
            while (free_[now_] == 0) ++now_;
            const int n = static_cast<int>(times < free_[now_] ? times : free_[now_]);
            const int end = std::min(now_ + d, slots_ - 1);
            free_[now_] -= n;
            free_[end] += n;
            times -= n;
            if (end > last_) last_ = end;
        }
    }
    double end() const { return static_cast<double>(last_) * unit_; }

private:
    static constexpr int kSlots = 4096;
    int unit_, slots_, now_ = 0, last_ = 0;
    int free_[kSlots];
};

// Raises the dynamic shared-memory limit of the forward kernel in a FwdMode once per device (b2a_fwd.cu).
int configure_fwd_kernel(const DeviceInfo& dev, int mode);

// Planner launch (b2a_plan.cu).  kind 0: forward items (256 query rows of a
// document, cost = visible key blocks).  kind 1: backward items (128 key rows
// of a document, cost = query tiles that see them).  Writes the whole workspace header.
int launch_varlen_plan(int kind, const int* cu_seqlens_q, const int* cu_seqlens_k, int batch,
                       int causal, int2* work_list, WorkspaceHeader* header, int max_entries_cap,
                       cudaStream_t stream);

// Optional per-thread kernel timing (b2a_profile_enable / b2a_profile_read).  The launchers
// call profile_mark(kind, false, stream) right before and profile_mark(kind, true, stream)
// right after the main kernel launch; both are no-ops unless profiling is enabled.
void profile_mark(int kernel, bool after, cudaStream_t stream);

}  // namespace b2a
