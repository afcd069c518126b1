// C-ABI entry point and launcher of the forward attention kernel.
#include "b2a_fwd.cuh"
#include "b2a_host.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace b2a {

namespace {

constexpr size_t kFwdSmemBytes = sizeof(FwdShared) + 1024;   // + slack for 1 KiB alignment

template <int kMode>
int set_fwd_smem_attribute() {
    B2A_CUDA_OK(cudaFuncSetAttribute(fwd_kernel<kMode>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kFwdSmemBytes)));
    return B2A_OK;
}

// log2 of the query heads that share a tile's rows: all heads of a K/V head's group where their number is a power of
// two that divides a tile (a TMA box of 128 / group rows of group heads is then one tile), none otherwise.  A tile of few
// query rows is mostly padding without it, and K and V are streamed once per head or pair of heads instead of once: one
// token for 16 sequences of 4,001, 32 over 8 heads, takes 46 us packed and 120 us not.  Full sequences take as long or a little
// less (4 x 2,048: 146 and 148 us, 1 x 32,768: 6,326 and 6,320 us), so there is no line between few and many rows.
int fwd_pack_shift(int heads_q, int heads_k) {
    const int group = heads_q / heads_k;
    if ((group & (group - 1)) != 0 || group > kTileM) return 0;
    int shift = 0;
    while ((1 << shift) < group) ++shift;
    return shift;
}

// How a fixed-length call is cut along its keys.  max_splits = 1: not at all.  The cut follows from the sizes and the
// device alone, so that a caller's own CTA count does not change the result.
struct FwdSplit {
    int max_splits = 1, whole_items = 0, blocks = 0, tiles = 0, rows = 0;
    long long items = 0;         // behind whole_items
    size_t stat_bytes = 0, o_bytes = 0;
    size_t total() const { return stat_bytes + o_bytes; }
};

// An item (up to 256 packed query rows against all keys they see) is the smallest thing a CTA takes.  Where there are
// few items, or they fill the CTAs unevenly, the keys are cut as well.  The cost of k pieces per item, in K/V blocks a
// CTA goes through (about 1.6 us each), is the number of rounds times the piece, plus one block a round for starting and
// storing a piece, three for the launch that adds up, and the time that writing and reading the pieces takes (6.8 MB in a
// block's time, about 4.2 TB/s: they stay in L2).  Where items differ a lot in length (a square causal call) the dynamic hand-out packs them,
// and the bound is the mean load plus half a piece.  A cut has to promise a twentieth: the model knows no better.
// That formula picks the number of pieces, but it holds half a piece against an uncut causal call too, whose shortest items
// come last and fill the gaps.  So the call is then handed out item by item both ways (HandOut), and again the cut has
// to promise a twentieth.
// Measured (us on the device, not cut / cut): 512 rows against 16,384 keys, 32 over 8 heads, two pieces: 194 / 114; 128 rows
// against 32,768: 375 / 69; 4 x 64 rows against 8,192: 101 / 46; 2 x 3,001 rows without a mask, 32 heads, the last of six
// rounds cut: 255 / 248.  Calls that this leaves alone, and what the formula's cut would make of them: 1 x 6,829 causal, 8 over
// 2 heads, 91 / 101; 1 x 6,192, 8 over 1, 84 / 91; 2 x 1,024, 16 over 4, 21 / 35; 16 x 1 row against 4,001, 45 / 58.  Groups
// that are no power of two are not packed, and their pairs of heads are not cut.
FwdSplit plan_fwd_split(const b2a_fwd_args& a, int ctas) {
    FwdSplit s;
    const int group = a.heads_q / a.heads_k;
    const int shift = fwd_pack_shift(a.heads_q, a.heads_k);
    if (a.cu_seqlens_q != nullptr || a.merge_running || a.prefetch_bytes != 0 || (1 << shift) != group) return s;
    const int rows = kFwdRowsPerWork >> shift;
    const long long pieces = (a.seqlen_q + rows - 1) / rows;
    const long long items = pieces * a.batch * a.heads_k;
    const int n = (a.seqlen_k + kTileN - 1) / kTileN;
    if (n < 8 || items >= 8ll * ctas) return s;
    const long long tile_rows = static_cast<long long>(a.seqlen_q) << shift;
    s.tiles = tile_rows > kTileM ? 2 : 1;
    s.rows = static_cast<int>(std::min<long long>(tile_rows, kTileM));
    auto blocks_of = [&](long long i) {   // that an item of piece i goes through
        const long long last = std::min<long long>((i + 1) * rows, a.seqlen_q);
        const long long limit = a.is_causal ? std::min<long long>(a.seqlen_k, last + a.seqlen_k - a.seqlen_q) : a.seqlen_k;
        return limit <= 0 ? 0 : static_cast<int>((limit + kTileN - 1) / kTileN);
    };
    double mean = 0;   // blocks of an item
    for (long long i = 0; i < pieces; ++i) mean += blocks_of(i);
    mean /= static_cast<double>(pieces);
    const bool even = mean > 0.8 * n;
    // Items of one length: only those of the last, incomplete round are cut.
    const long long whole = even ? items / ctas * ctas : 0;
    const double cut = static_cast<double>(items - whole);
    if (cut == 0) return FwdSplit{};
    const double piece_bytes = 2.0 * s.tiles * s.rows * (kHeadDim + 2) * sizeof(float);   // written and read
    auto cost = [&](int k) {
        const double piece = (n + k - 1) / k, extra = k > 1 ? 1.0 : 0.0, add = k > 1 ? 3.0 + cut * k * piece_bytes / 6.8e6 : 0.0;
        const double load = cut * k / ctas;
        if (even) return static_cast<double>(whole / ctas) * n + std::ceil(load) * (piece + extra) + add;
        return std::max(piece, cut * mean / ctas) + 0.5 * piece + extra * load + add;
    };
    int best = 1;
    for (int k = 2; k <= kFwdMaxSplits && n / k >= 4; ++k) {
        if (cost(k) < cost(best)) best = k;
    }
    if (best == 1 || cost(best) > 0.95 * cost(1)) return FwdSplit{};
    s.whole_items = static_cast<int>(whole);
    s.max_splits = best;
    s.blocks = (n + best - 1) / best;
    s.items = items - whole;
    // The same two calls handed out item by item.
    const double steps = mean * items + 3.0 * items * best;
    HandOut uncut(ctas, steps, n + 2), pieced(ctas, steps, n + 2);
    long long left_whole = whole, parts_cut = 0;
    for (int b = 0; b < a.batch; ++b) {
        for (long long i = 0; i < pieces; ++i) {
            const int blocks = blocks_of(a.is_causal ? pieces - 1 - i : i);
            const long long first = std::min<long long>(left_whole, a.heads_k), rest = a.heads_k - first;
            const int k = std::min(best, std::max(1, (blocks + s.blocks - 1) / s.blocks));
            uncut.add(blocks + 1, a.heads_k);
            pieced.add(blocks + 1, first);
            pieced.add((blocks + k - 1) / k + 1 + (k > 1 ? 1 : 0), rest * k);
            left_whole -= first;
            if (k > 1) parts_cut += rest * k;
        }
    }
    if (pieced.end() + 3.0 + parts_cut * piece_bytes / 6.8e6 > 0.95 * uncut.end()) return FwdSplit{};
    const size_t parts = static_cast<size_t>(cut) * best * s.tiles;
    s.stat_bytes = align_up(parts * s.rows * sizeof(float2), 256);
    s.o_bytes = align_up(parts * s.rows * kHeadDim * sizeof(float), 256);
    return s.total() > (128ull << 20) ? FwdSplit{} : s;   // callers allocate it for every call
}

// ---------------------------------------------------------------------------------------
// Adds up the pieces of a key split, in the order of their keys: O = sum_i w_i O_i / sum_i w_i l_i with
// w_i = 2^(m_i - max m).  One CTA per 32 rows of a tile, a kernel of its own: bound by reading the pieces
// (512 bytes per row and piece, from L2), which takes the whole chip; left to the CTA that finishes an item last,
// the same sum was a chain of L2 latencies longer than most items (24 us more on a call of 40 us).
// ---------------------------------------------------------------------------------------
constexpr int kCombineRows = 32;

__global__ void __launch_bounds__(256)
fwd_combine_kernel(const FwdParams p) {
    constexpr int kPitch = kHeadDim + 4;    // bf16; keeps the 8-byte column stores of 16 rows on distinct banks
    __shared__ __align__(8) __nv_bfloat16 out[kCombineRows * kPitch];
    __shared__ float weight[kFwdMaxSplits][kCombineRows];
    let_next_kernel_start();
    wait_for_previous_kernel();
    const int strips = (p.split_rows + kCombineRows - 1) / kCombineRows;
    const int strip = blockIdx.x % strips;
    const int x = blockIdx.x / strips % p.split_tiles;
    const int item = blockIdx.x / (strips * p.split_tiles);
    const int w = p.whole_items + item * p.max_splits;
    const FwdWork wk = fwd_decode_work<true>(p, w, w + 1);
    const int row0 = fwd_tile_row0(wk, x);
    const int first = strip * kCombineRows;                                        // of the tile's rows
    const int rows = min(min(kCombineRows, p.split_rows - first), ((wk.q_len - row0) << wk.shift) - first);
    if (wk.splits == 1 || rows <= 0) return;
    const long long step = static_cast<long long>(p.split_tiles) * p.split_rows;   // rows from piece to piece
    const long long at = static_cast<long long>(item) * p.max_splits * step + x * p.split_rows + first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int head0 = fwd_tile_head(wk, x);
    // What the uncut kernel leaves of NaN and infinities is left here as well: a sum that is NaN or empty gives the norm 0
    // (O * 0 keeps NaN) and -inf for LSE, and a piece whose weight is 0 is multiplied by it like the others.  Only a
    // piece without a block for this tile is skipped (sum -1, weight -1): its O was never stored.
    if (warp == 0 && lane < rows) {
        float m = -INFINITY, l = 0.f;
        for (int i = 0; i < wk.splits; ++i) m = fmaxf(m, p.split_stat[at + i * step + lane].x);
        for (int i = 0; i < wk.splits; ++i) {
            const float2 st = p.split_stat[at + i * step + lane];
            // -inf: the row saw no key here (or only NaN, which its sum carries).  m itself may be infinite.
            const float f = st.x == -INFINITY ? 0.f : st.x == m ? 1.f : fast_exp2((st.x - m) * p.scale_log2);
            const bool stored = st.y != -1.f;
            weight[i][lane] = stored ? f : -1.f;
            if (stored) l = fmaf(st.y, f, l);
        }
        const bool seen = l > 0.f && m != -INFINITY;
        const float norm = seen ? 1.f / l : 0.f;
        for (int i = 0; i < wk.splits; ++i) {
            const float f = weight[i][lane];
            if (f != -1.f) weight[i][lane] = f * norm;
        }
        const int tr = first + lane;
        p.lse[wk.lse_base + static_cast<long long>(head0 - wk.head + (tr & ((1 << wk.shift) - 1))) * p.lse_head_stride + row0 +
              (tr >> wk.shift)] = seen ? (m * p.scale_log2 + fast_log2(l)) * kLn2 : -INFINITY;
    }
    __syncthreads();
    // Lane = row, four of the 32 column quads a warp.
    if (lane < rows) {
        const long long base = (static_cast<long long>(item) * p.max_splits * step + x * p.split_rows) * 32 + first + lane;
        float4 acc[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
        for (int i = 0; i < wk.splits; ++i) {
            const float f = weight[i][lane];
            if (f == -1.f) continue;
            const float4* o = p.split_o + base + i * step * 32;
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = __ldcs(o + static_cast<long long>(warp * 4 + u) * p.split_rows);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                acc[u].x = fmaf(v[u].x, f, acc[u].x);
                acc[u].y = fmaf(v[u].y, f, acc[u].y);
                acc[u].z = fmaf(v[u].z, f, acc[u].z);
                acc[u].w = fmaf(v[u].w, f, acc[u].w);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            *reinterpret_cast<uint2*>(&out[lane * kPitch + (warp * 4 + u) * 4]) =
                make_uint2(pack_bf16x2(acc[u].x, acc[u].y), pack_bf16x2(acc[u].z, acc[u].w));
        }
    }
    __syncthreads();
    // A warp writes one whole 256-byte row per instruction.
    for (int rr = warp; rr < rows; rr += 8) {
        const int tr = first + rr;
        const long long to = (static_cast<long long>(wk.q_begin) + row0 + (tr >> wk.shift)) * p.heads_q + head0 +
                             (tr & ((1 << wk.shift) - 1));
        *reinterpret_cast<uint2*>(p.o + to * kHeadDim + lane * 4) = *reinterpret_cast<const uint2*>(&out[rr * kPitch + lane * 4]);
    }
}

}  // namespace

int configure_fwd_kernel(const DeviceInfo& dev, int mode) {
    if (static_cast<size_t>(dev.max_smem_optin) < kFwdSmemBytes) {
        return fail(B2A_ERR_UNSUPPORTED_DEVICE, "device offers %d bytes of shared memory, need %zu",
                    dev.max_smem_optin, kFwdSmemBytes);
    }
    return mode == kFwdMerge   ? once_per_device(dev.device, 1, set_fwd_smem_attribute<kFwdMerge>)
           : mode == kFwdSplit ? once_per_device(dev.device, 4, set_fwd_smem_attribute<kFwdSplit>)
                               : once_per_device(dev.device, 0, set_fwd_smem_attribute<kFwdPlain>);
}

}  // namespace b2a

extern "C" {

size_t b2a_fwd_workspace_bytes(int32_t batch, int32_t total_q, int32_t is_varlen) {
    const size_t behind = is_varlen ? b2a::max_entries(batch, total_q, b2a::kFwdRowsPerWork) * sizeof(int2)
                                    : b2a::kFwdStatusWords * sizeof(unsigned int);
    return b2a::align_up(sizeof(b2a::WorkspaceHeader) + behind, 256);
}

size_t b2a_fwd_scratch_bytes(const b2a_fwd_args* a) {
    using namespace b2a;
    if (a == nullptr) return 0;
    const size_t need = b2a_fwd_workspace_bytes(a->batch, a->total_q, a->cu_seqlens_q != nullptr ? 1 : 0);
    DeviceInfo dev{};
    if (a->batch < 1 || a->heads_q < 1 || a->heads_k < 1 || a->heads_q % a->heads_k != 0 || a->seqlen_q < 1 ||
        a->seqlen_k < 1 || current_device_info(&dev) != B2A_OK) {
        return need;   // b2a_fwd reports what is wrong
    }
    const size_t split = plan_fwd_split(*a, dev.sm_count).total();
    return split > 0 ? need + split : need;
}

int b2a_fwd(const b2a_fwd_args* a, void* cuda_stream) {
    using namespace b2a;
    if (a == nullptr || a->workspace == nullptr) return b2a_fwd_with_scratch(a, nullptr, 0, cuda_stream);
    const size_t need = b2a_fwd_workspace_bytes(a->batch, a->total_q, a->cu_seqlens_q != nullptr ? 1 : 0);
    if (a->workspace_bytes <= need) return b2a_fwd_with_scratch(a, nullptr, 0, cuda_stream);
    return b2a_fwd_with_scratch(a, static_cast<uint8_t*>(a->workspace) + need, a->workspace_bytes - need, cuda_stream);
}

int b2a_fwd_with_scratch(const b2a_fwd_args* a, void* scratch, size_t scratch_bytes, void* cuda_stream) {
    using namespace b2a;
    B2A_REQUIRE(a != nullptr, "args must not be NULL");
    B2A_REQUIRE(a->q && a->k && a->v && a->out && a->lse, "q, k, v, out and lse must not be NULL");
    B2A_REQUIRE(a->head_dim == kHeadDim, "head_dim must be 128, got %d", a->head_dim);
    B2A_REQUIRE(a->batch >= 1, "batch must be >= 1, got %d", a->batch);
    B2A_REQUIRE(a->heads_q >= 1 && a->heads_k >= 1 && a->heads_q % a->heads_k == 0,
                "heads_q %% heads_k must be 0, got heads_q=%d heads_k=%d", a->heads_q, a->heads_k);
    B2A_REQUIRE(a->total_q >= 1 && a->total_k >= 1, "total_q and total_k must be positive");
    B2A_REQUIRE((a->cu_seqlens_q == nullptr) == (a->cu_seqlens_k == nullptr),
                "cu_seqlens_q and cu_seqlens_k must both be given or both be NULL");
    const bool varlen = a->cu_seqlens_q != nullptr;
    if (!varlen) {
        B2A_REQUIRE(a->seqlen_q >= 1 && a->seqlen_k >= 1, "seqlen_q and seqlen_k must be positive");
        B2A_REQUIRE(static_cast<long long>(a->batch) * a->seqlen_q == a->total_q &&
                        static_cast<long long>(a->batch) * a->seqlen_k == a->total_k,
                    "BSHD sizes must satisfy total = batch * seqlen");
    }
    B2A_REQUIRE(a->grid_blocks >= 0, "grid_blocks must be >= 0, got %d", a->grid_blocks);
    const bool prefetch = a->prefetch_bytes != 0;
    if (prefetch) {
        B2A_REQUIRE(a->prefetch_src_k && a->prefetch_src_v && a->prefetch_dst_k && a->prefetch_dst_v,
                    "prefetch source and destination pointers must not be NULL when prefetch_bytes > 0");
        B2A_REQUIRE(a->prefetch_bytes % 16 == 0, "prefetch_bytes must be a multiple of 16, got %zu", a->prefetch_bytes);
        B2A_REQUIRE(a->prefetch_blocks > 0, "prefetch_blocks must be positive when prefetch_bytes > 0, got %d",
                    a->prefetch_blocks);
        const uintptr_t align = reinterpret_cast<uintptr_t>(a->prefetch_src_k) | reinterpret_cast<uintptr_t>(a->prefetch_src_v) |
                                reinterpret_cast<uintptr_t>(a->prefetch_dst_k) | reinterpret_cast<uintptr_t>(a->prefetch_dst_v);
        B2A_REQUIRE((align & 0xF) == 0, "prefetch buffers must be 16-byte aligned");
    }
    B2A_REQUIRE(a->workspace != nullptr && (reinterpret_cast<uintptr_t>(a->workspace) & 0xF) == 0,
                "workspace must be a 16-byte aligned device pointer");
    B2A_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 0xF) == 0, "scratch must be 16-byte aligned");
    const size_t need = b2a_fwd_workspace_bytes(a->batch, a->total_q, varlen ? 1 : 0);
    // A fixed-length call without room for a status word per CTA runs all the same, with the counter.
    const size_t least = varlen ? need : align_up(sizeof(WorkspaceHeader), 256);
    if (a->workspace_bytes < least) {
        return fail(B2A_ERR_WORKSPACE_TOO_SMALL, "workspace has %zu bytes, need %zu",
                    a->workspace_bytes, need);
    }

    DeviceInfo dev{};
    int rc = current_device_info(&dev);
    if (rc != B2A_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);

    const int pack_shift = fwd_pack_shift(a->heads_q, a->heads_k);
    CUtensorMap map_q, map_k, map_v;
    rc = make_token_map(&map_q, a->q, a->total_q, a->heads_q, kTileM >> pack_shift, 1u << pack_shift);
    if (rc != B2A_OK) return rc;
    rc = make_token_map(&map_k, a->k, a->total_k, a->heads_k, kTileN);
    if (rc != B2A_OK) return rc;
    rc = make_token_map(&map_v, a->v, a->total_k, a->heads_k, kTileN);
    if (rc != B2A_OK) return rc;

    auto* hdr = static_cast<WorkspaceHeader*>(a->workspace);
    int2* work_list = reinterpret_cast<int2*>(hdr + 1);
    FwdSplit split;
    if (scratch != nullptr && scratch_bytes > 0) split = plan_fwd_split(*a, dev.sm_count);
    if (scratch_bytes < split.total()) split = FwdSplit{};   // b2a_fwd_workspace_bytes is enough to run
    uint8_t* split_ws = static_cast<uint8_t*>(scratch);

    FwdParams p{};
    p.o = static_cast<__nv_bfloat16*>(a->out);
    p.lse = a->lse;
    p.cu_seqlens_q = a->cu_seqlens_q;
    p.cu_seqlens_k = a->cu_seqlens_k;
    p.work_list = varlen ? work_list : nullptr;
    p.num_entries_dev = &hdr->num_entries;
    p.sched_counter = &hdr->sched_counter;
    p.status = &hdr->status;
    p.batch = a->batch;
    p.seqlen_q = a->seqlen_q;
    p.seqlen_k = a->seqlen_k;
    p.total_q = a->total_q;
    p.total_k = a->total_k;
    p.heads_q = a->heads_q;
    p.heads_k = a->heads_k;
    p.causal = a->is_causal ? 1 : 0;
    p.scale = a->softmax_scale > 0.f ? a->softmax_scale : 1.0f / std::sqrt(static_cast<float>(kHeadDim));
    p.scale_log2 = p.scale * kLog2e;
    p.merge = a->merge_running ? 1 : 0;
    p.timeout_ns = wait_timeout_ns();
    p.pack_shift = pack_shift;
    p.max_splits = split.max_splits;
    p.whole_items = split.whole_items;
    p.split_blocks = split.blocks;
    p.split_tiles = split.tiles;
    p.split_rows = split.rows;
    p.split_stat = reinterpret_cast<float2*>(split_ws);
    p.split_o = reinterpret_cast<float4*>(split_ws + split.stat_bytes);

    long long work_items;
    if (varlen) {
        const int cap = static_cast<int>(max_entries(a->batch, a->total_q, kFwdRowsPerWork));
        rc = launch_varlen_plan(0, a->cu_seqlens_q, a->cu_seqlens_k, a->batch, p.causal, work_list,
                                hdr, cap, stream);
        if (rc != B2A_OK) return rc;
        p.num_entries_host = cap;
        p.lse_head_stride = a->total_q;
        p.lse_batch_stride = 0;
        work_items = static_cast<long long>(cap) * a->heads_q;
    } else {
        const int rows = kFwdRowsPerWork >> pack_shift;
        const int nmb = (a->seqlen_q + rows - 1) / rows;
        p.num_entries_host = a->batch * nmb;
        p.lse_head_stride = a->seqlen_q;
        p.lse_batch_stride = static_cast<long long>(a->heads_q) * a->seqlen_q;
        work_items = static_cast<long long>(p.num_entries_host) * fwd_items_per_entry(p);
        work_items += (work_items - p.whole_items) * (p.max_splits - 1);
    }

    int grid = a->grid_blocks > 0 ? a->grid_blocks : dev.sm_count;
    // Packed documents: the planner writes the header.  One item a CTA and a status word for each: the kernel does.  Else a memset,
    // a launch more: 2 to 3 us of a call that takes 9 (1 x 128, 32 heads) to 60.
    if (!varlen && work_items <= std::min(grid, dev.sm_count) && a->workspace_bytes >= need &&
        work_items + (prefetch ? a->prefetch_blocks : 0) <= kFwdStatusWords) {
        p.sched_counter = nullptr;
        p.status = reinterpret_cast<unsigned int*>(hdr + 1);
        p.status_step = 1u;
    } else if (!varlen) {
        B2A_CUDA_OK(cudaMemsetAsync(hdr, 0, sizeof(WorkspaceHeader), stream));
    }
    if (work_items < grid) grid = static_cast<int>(work_items);
    if (grid < 1) grid = 1;
    p.num_comp = grid;
    if (prefetch) {
        // Copy CTAs ride in the same launch behind the compute CTAs; neither kind waits for the other.
        p.prefetch_src[0] = static_cast<const uint8_t*>(a->prefetch_src_k);
        p.prefetch_src[1] = static_cast<const uint8_t*>(a->prefetch_src_v);
        p.prefetch_dst[0] = static_cast<uint8_t*>(a->prefetch_dst_k);
        p.prefetch_dst[1] = static_cast<uint8_t*>(a->prefetch_dst_v);
        p.prefetch_bytes = a->prefetch_bytes;
        grid += a->prefetch_blocks;
    }

    const int mode = p.merge ? kFwdMerge : p.max_splits > 1 ? kFwdSplit : kFwdPlain;
    rc = configure_fwd_kernel(dev, mode);
    if (rc != B2A_OK) return rc;
    profile_mark(B2A_KERNEL_FWD, false, stream);
    if (mode == kFwdMerge) {
        B2A_CUDA_OK(launch_early(fwd_kernel<kFwdMerge>, grid, kFwdThreads, kFwdSmemBytes, stream, map_q, map_k, map_v, p));
    } else if (mode == kFwdSplit) {
        B2A_CUDA_OK(launch_early(fwd_kernel<kFwdSplit>, grid, kFwdThreads, kFwdSmemBytes, stream, map_q, map_k, map_v, p));
    } else {
        B2A_CUDA_OK(launch_early(fwd_kernel<kFwdPlain>, grid, kFwdThreads, kFwdSmemBytes, stream, map_q, map_k, map_v, p));
    }
    if (mode == kFwdSplit) {
        const long long strips = static_cast<long long>(split.items) * split.tiles * ((split.rows + kCombineRows - 1) / kCombineRows);
        B2A_CUDA_OK(launch_early(fwd_combine_kernel, static_cast<unsigned int>(strips), 256, 0, stream, p));
    }
    profile_mark(B2A_KERNEL_FWD, true, stream);
    B2A_CUDA_OK(cudaGetLastError());
    return B2A_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Forward for callers that cannot allocate device memory
// ---------------------------------------------------------------------------------------
namespace b2a {
namespace {

// Scratch of b2a_fwd_noalloc: the 16-byte workspace header plus the varlen work list.
// 64 KiB holds 8190 work pieces (a piece is 256 query rows of one document), i.e. packed
// batches with total_q / 256 + batch + 1 <= 8190.  Every GPU that loads the library keeps
// this array resident until the process exits.
constexpr size_t kNoAllocScratchBytes = 64 * 1024;
static __device__ __align__(256) unsigned char g_fwd_noalloc_scratch[kNoAllocScratchBytes];

}  // namespace

// Device address of the array on each device.  The array's name is only a host-side handle
// in host code; the address a kernel can use comes from cudaGetSymbolAddress, asked once per
// device while that device is current.
int noalloc_scratch_ptr(void** out) {
    static std::mutex mu;
    static void* ptrs[64] = {};
    int dev = 0;
    B2A_CUDA_OK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        return fail(B2A_ERR_CUDA, "device index %d out of range", dev);
    }
    std::lock_guard<std::mutex> lock(mu);
    if (ptrs[dev] == nullptr) {
        void* p = nullptr;
        cudaError_t err = cudaGetSymbolAddress(&p, g_fwd_noalloc_scratch);
        if (err != cudaSuccess || p == nullptr) {
            return fail(B2A_ERR_CUDA, "cudaGetSymbolAddress(scratch) failed on device %d: %s", dev,
                        cudaGetErrorString(err));
        }
        ptrs[dev] = p;
    }
    *out = ptrs[dev];
    return B2A_OK;
}

}  // namespace b2a

extern "C" {

size_t b2a_fwd_noalloc_scratch_limit(void) { return b2a::kNoAllocScratchBytes; }

int b2a_fwd_noalloc(const b2a_fwd_args* a, void* cuda_stream) {
    using namespace b2a;
    B2A_REQUIRE(a != nullptr, "args must not be NULL");
    B2A_REQUIRE(a->batch >= 1 && a->total_q >= 1, "batch and total_q must be positive");
    const bool varlen = a->cu_seqlens_q != nullptr;
    const size_t need = b2a_fwd_workspace_bytes(a->batch, a->total_q, varlen ? 1 : 0);
    if (need > kNoAllocScratchBytes) {
        return fail(B2A_ERR_WORKSPACE_TOO_SMALL,
                    "b2a_fwd_noalloc: this problem needs %zu bytes of scratch but the built-in scratch "
                    "holds %zu (packed batches up to total_q / 256 + batch + 1 <= 8190); "
                    "use b2a_fwd with a caller-provided workspace",
                    need, kNoAllocScratchBytes);
    }
    void* scratch = nullptr;
    int rc = noalloc_scratch_ptr(&scratch);
    if (rc != B2A_OK) return rc;
    b2a_fwd_args local = *a;
    local.workspace = scratch;
    local.workspace_bytes = need;   // never enough for a key split: the array holds no partial results
    return b2a_fwd(&local, cuda_stream);
}

}  // extern "C"
