// MoE pipelines as ONE host call each: align -> quantise -> grouped GEMM1 with fused SiLU*up -> quantise ->
// grouped GEMM2 with the router weight (-> top-k sum), issued back to back from C++ into a caller's
// workspace.
//
// Two orders of the rows between the launches:
//   gathered  (few rows per expert: decode) the GEMMs fetch their A rows through sorted_ids with
//             tile::gather4 and store in route-slot order: nothing touches padding rows.  The copy into
//             expert order and the padding cost 60 us of a 32-token DeepSeek-V3 step.
//   sorted    (otherwise) rows are laid out in expert order, padded to 128 per expert (256 where CTA pairs run
//             the products), and fetched as TMA boxes.  Padding rows are zeros all the way: written once,
//             they cost less than the tensor power that stale bytes in their place draw (2 % of a step
//             under the power cap).  A gather4 of four 128-byte rows takes ~70 cycles whatever the rows, so
//             a full tile of them (32 per K block) is four times slower than its MMAs: the line lies
//             where eight lanes' gathers still hide behind the weight stream (use_gather).
#include <mutex>

#include "common.cuh"

// Built-in scratch of fg_moe_routed_block_fp8_local_noalloc: part of the library image, so every
// GPU on which the library is loaded keeps these bytes reserved until the process exits.
// In host code this name is only a handle for cudaGetSymbolAddress, never a device address.
static __device__ __align__(256) unsigned char g_routed_scratch[FG_NOALLOC_SCRATCH_BYTES];

namespace {

constexpr int TILE_ROWS = 128;
constexpr int PAIR_ROWS = 256;      // rows of a CTA pair's tile
constexpr int PAIR_MIN_ROWS = 768;  // rows per expert from which pairs are used (see use_pairs)

inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// What an expert pipeline keeps between its launches.
struct Workspace {
    int32_t* sorted_ids;
    int32_t* expert_ids;
    int32_t* post_pad;
    float* scalars;  // per-tensor modes: amax and scale of both GEMMs' inputs; 16-bit mode: unit scales
    uint8_t* a1;     // input rows of GEMM1: quantised, or 16-bit copies in expert order
    float* a1s;
    uint8_t* act;    // GEMM1's output
    uint8_t* a2;     // the same quantised
    float* a2s;
    uint8_t* routed; // GEMM2's output, one row per route slot
    int64_t max_pad, n_blocks, rows, bytes;
};

struct Carver {
    uint8_t* p;
    int64_t off;
    uint8_t* take(int64_t bytes) {
        uint8_t* r = p ? p + off : nullptr;
        off += align_up(bytes, 256);
        return r;
    }
};

// Sorted rows of `slots` route slots: every expert padded to the tile, and no more than one tile per slot.
void carve_tables(Carver& c, Workspace& w, int64_t slots, int num_experts, int tile = TILE_ROWS) {
    w.max_pad = slots + (int64_t)num_experts * (tile - 1);
    if (slots * tile < w.max_pad) w.max_pad = slots * tile;
    w.n_blocks = fg_cdiv(w.max_pad, tile);
    w.rows = w.max_pad / tile * tile;
    w.sorted_ids = (int32_t*)c.take(4 * w.max_pad);
    w.expert_ids = (int32_t*)c.take(4 * w.n_blocks);
    w.post_pad = (int32_t*)c.take(256);
}

// Routed block-FP8 pipeline.
Workspace carve(void* base, int64_t slots, int num_experts, int64_t H, int64_t I, int esz) {
    Workspace w{};
    Carver c{reinterpret_cast<uint8_t*>(base), 0};
    carve_tables(c, w, slots, num_experts);
    w.a1 = c.take(w.rows * H);
    w.a1s = (float*)c.take(4 * w.rows * (H / 128));
    w.act = c.take(w.rows * I * esz);
    w.a2 = c.take(w.rows * I);
    w.a2s = (float*)c.take(4 * w.rows * (I / 128));
    w.bytes = c.off;
    return w;
}

int check_dims(int64_t n_in, int num_experts, int64_t H, int64_t I, int out_dtype) {
    FG_REQUIRE(n_in >= 0 && num_experts > 0 && H > 0 && I > 0, FG_ERR_INVALID_ARGUMENT, "bad sizes");
    FG_REQUIRE(H % 128 == 0 && I % 128 == 0, FG_ERR_UNSUPPORTED,
               "hidden %lld and intermediate %lld must be multiples of 128", (long long)H, (long long)I);
    FG_REQUIRE(out_dtype == FG_DTYPE_BF16 || out_dtype == FG_DTYPE_F16, FG_ERR_UNSUPPORTED,
               "activations must be bf16 or fp16");
    return FG_OK;
}

// One layer's experts on tokens of this GPU.
struct Experts {
    int mode;
    const void* hidden;
    int dtype;
    const void* topk_w;
    int topk_w_dtype;
    int64_t T;
    int topk;
    const void *w1, *w2;
    const float *s1, *s2, *a1_scale, *a2_scale;
    int local_experts;
    int64_t H, I;
    bool gathered, pairs;
};

// Whether rows in expert order are padded to 256 per expert instead of 128 and the products run by CTA pairs:
// `slots` rows against outputs of n1 and n2 columns.  A pair moves a third fewer operand bytes per flop and
// pays 64 more padding rows per expert on average.  Steady state under the power cap, single -> pair: Mixtral,
// 1024 rows per expert: fp8 1620 -> 1518 us, int8 1532 -> 1390, bf16 2875 -> 2710; 1024 rows per group x 4096 x 7168:
// 256 -> 242; but 525 rows per expert: 984 -> 990, 500 rows per group x 4096 x 4096: 84.5 -> 89.  Hence 768
// rows per expert, and three waves of pair tiles in the smaller product.
bool use_pairs(int64_t slots, int num_experts, int64_t n1, int64_t n2) {
    const int64_t n = n1 < n2 ? n1 : n2;
    return slots >= PAIR_MIN_ROWS * (int64_t)num_experts && slots / PAIR_ROWS * (n / 256) >= 3 * (int64_t)(fg_num_sms() / 2);
}

// The line between the two row orders (see the head of this file): 32 rows per expert, or 16 where the experts are
// many.  A large router is skewed, and its popular experts then have full tiles of gathered rows long before
// the average says so.  Gathered / sorted, us per step: DeepSeek-V3 (256 experts) 12 rows per expert
// 2048 / 2101, 28 rows 2485 / 2356; Mixtral (8) 12 rows 260 / 280, 30 rows 277 / 282.
bool use_gather(int64_t slots, int num_experts) { return slots <= (num_experts > 32 ? 16 : 32) * (int64_t)num_experts; }

// Rows of one GEMM's input in the operand type of the mode; *scale is where their scales are.  `slots` (NULL or the
// alignment table): only the rows that it names count toward a dynamic per-tensor scale.  In route-slot
// order a slot whose expert id is out of range has a row that nothing wrote.
int quantise(int mode, const void* x, int dtype, uint8_t* q, float* s, float* scalars, const float* given, int64_t src_rows,
             int64_t rows, int64_t K, const int32_t* index, int div, int64_t limit, const int32_t* n_rows_dev, const float** scale,
             cudaStream_t st, const Workspace* slots = nullptr) {
    *scale = s;
    const int kind = mode == FG_EXPERTS_BLOCK_FP8 ? FG_QUANT_GROUP128 : mode == FG_EXPERTS_CHANNEL_FP8 ? FG_QUANT_TOKEN
                     : mode == FG_EXPERTS_CHANNEL_INT8 ? FG_QUANT_INT8 : FG_QUANT_TENSOR;
    const float* tensor = given;
    if (kind == FG_QUANT_TENSOR) {
        *scale = given ? given : scalars + 1;
        if (!given) {  // scalars[0]: amax, scalars[1]: the scale derived from it
            FG_CUDA(cudaMemsetAsync(scalars, 0, 4, st));
            const int rc = slots ? fg_abs_max_rows(x, dtype, slots->max_pad, K, K, slots->post_pad, slots->sorted_ids, (int32_t)src_rows,
                                                   scalars, st)
                                 : fg_abs_max(x, dtype, src_rows, K, K, index && div == 0 ? n_rows_dev : nullptr, scalars, st);
            if (rc != FG_OK) return rc;
            tensor = scalars;
        }
    }
    return fg_quant_rows(kind, x, dtype, q, s, tensor, given ? nullptr : scalars + 1, rows, K, index, div, (int32_t)limit,
                         n_rows_dev, st);
}

// align has run: quantise -> GEMM1 -> quantise -> GEMM2 into y (route-slot order).
int run_experts(const Experts& e, const Workspace& ws, void* y, cudaStream_t st) {
    const int64_t slots = e.T * e.topk;
    const bool unit = e.mode == FG_EXPERTS_16BIT, plain = unit || e.mode == FG_EXPERTS_16BIT_SCALED;
    const bool block = e.mode == FG_EXPERTS_BLOCK_FP8, tensor = e.mode == FG_EXPERTS_TENSOR_FP8;
    const int esz = e.dtype == FG_DTYPE_F32 ? 4 : 2;
    const void *a1 = ws.a1, *a2 = ws.a2;
    const float *a1s = ws.a1s, *a2s = ws.a2s, *s1 = e.s1, *s2 = e.s2;
    int rc = FG_OK;
    if (plain) {
        // unquantised activations: unit scales, per expert or (with scaled weights) per row
        float* ones = unit ? ws.scalars : ws.a1s;
        rc = fg_fill_ones(ones, unit ? e.local_experts : ws.rows, st);
        if (rc != FG_OK) return rc;
        a1s = a2s = ones;
        if (unit) s1 = s2 = ones;
        a2 = ws.act;
        if (e.gathered) a1 = e.hidden;
        else rc = fg_gather_rows_fp8(e.hidden, nullptr, ws.a1, nullptr, ws.rows, 2 * e.H, 0, 2 * e.H, 1, ws.sorted_ids, e.topk,
                                 (int32_t)slots, ws.post_pad, st);
    } else if (e.gathered) {
        rc = quantise(e.mode, e.hidden, e.dtype, ws.a1, ws.a1s, ws.scalars, e.a1_scale, e.T, e.T, e.H, nullptr, 1, 0, nullptr, &a1s, st);
    } else {
        // Each token is quantised once and its row copied to its top-k places; with one or two places
        // quantising while copying moves no more bytes and saves the launch.  The token rows borrow the
        // room of GEMM1's output, which is first written after the copy has finished.
        const int64_t s_cols = block ? e.H / 128 : 1, tok_q_bytes = align_up(e.T * e.H, 256);
        if (e.topk > 2 && !tensor && tok_q_bytes + 4 * e.T * s_cols <= ws.rows * e.I * esz) {
            uint8_t* tok_q = ws.act;
            float* tok_s = reinterpret_cast<float*>(ws.act + tok_q_bytes);
            rc = quantise(e.mode, e.hidden, e.dtype, tok_q, tok_s, ws.scalars, nullptr, e.T, e.T, e.H, nullptr, 1, 0, nullptr, &a1s, st);
            if (rc != FG_OK) return rc;
            a1s = ws.a1s;
            rc = fg_gather_rows_fp8(tok_q, tok_s, ws.a1, ws.a1s, ws.rows, e.H, s_cols, e.H, s_cols, ws.sorted_ids, e.topk, (int32_t)slots,
                                ws.post_pad, st);
        } else {
            rc = quantise(e.mode, e.hidden, e.dtype, ws.a1, ws.a1s, ws.scalars, e.a1_scale, e.T, ws.rows, e.H, ws.sorted_ids, e.topk,
                          slots, ws.post_pad, &a1s, st);
        }
    }
    if (rc != FG_OK) return rc;

    FgGroupedGemm g{};
    g.sorted_ids = ws.sorted_ids; g.expert_ids = ws.expert_ids; g.num_post_pad = ws.post_pad; g.max_rows = ws.rows;
    g.numel = slots; g.num_experts = e.local_experts; g.block_rows = e.pairs ? PAIR_ROWS : TILE_ROWS; g.cta_pairs = e.pairs;
    g.out_dtype = e.dtype;
    g.operand = plain ? (e.dtype == FG_DTYPE_BF16 ? 2 : 3) : e.mode == FG_EXPERTS_CHANNEL_INT8 ? 1 : 0;
    g.scale_mode = block ? FG_SCALE_BLOCK : (unit || tensor) ? FG_SCALE_SCALAR : FG_SCALE_VECTOR;
    g.c = ws.act; g.a = a1; g.w = e.w1; g.a_scale = a1s; g.w_scale = s1; g.a_rows = e.T; g.gather_div = e.gathered ? e.topk : 0;
    g.N = 2 * e.I; g.K = e.H; g.ld_a = e.H; g.ld_as = e.H / 128; g.ld_c = e.I; g.fuse_silu = 1; g.scatter = e.gathered;
    rc = fg_grouped_gemm(g, st);
    if (rc != FG_OK) return rc;
    if (!plain) {
        if (e.gathered) rc = quantise(e.mode, ws.act, e.dtype, ws.a2, ws.a2s, ws.scalars + 2, e.a2_scale, slots, slots, e.I, nullptr, 1,
                                      0, nullptr, &a2s, st, &ws);
        else rc = quantise(e.mode, ws.act, e.dtype, ws.a2, ws.a2s, ws.scalars + 2, e.a2_scale, ws.rows, ws.rows, e.I, ws.sorted_ids, 0,
                           slots, ws.post_pad, &a2s, st);
        if (rc != FG_OK) return rc;
    }
    g.c = y; g.a = a2; g.w = e.w2; g.a_scale = a2s; g.w_scale = s2; g.a_rows = slots; g.gather_div = e.gathered ? 1 : 0;
    g.N = e.H; g.K = e.I; g.ld_a = e.I; g.ld_as = e.I / 128; g.ld_c = e.H; g.fuse_silu = 0; g.scatter = 1; g.mul_weight = 1;
    g.topk_w = e.topk_w; g.topk_w_dtype = e.topk_w_dtype; g.topk_w_stride = 1;
    return fg_grouped_gemm(g, st);
}

// Device address of g_routed_scratch on the current device, looked up once per device.
int builtin_scratch(void** out) {
    static std::mutex mu;
    static void* addr[64] = {nullptr};
    int dev = -1;
    FG_CUDA(cudaGetDevice(&dev));
    FG_REQUIRE(dev >= 0 && dev < 64, FG_ERR_UNSUPPORTED, "device index %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        FG_CUDA(cudaGetSymbolAddress((void**)&p, g_routed_scratch));
        addr[dev] = p;
    }
    *out = addr[dev];
    return FG_OK;
}

}  // namespace

namespace {

// Scratch of fg_scaled_grouped_mm_fp8: the alignment tables only.
Workspace carve_grouped_mm(void* base, int64_t m_total, int num_groups, int tile) {
    Workspace w{};
    Carver c{reinterpret_cast<uint8_t*>(base), 0};
    carve_tables(c, w, m_total, num_groups, tile);
    w.bytes = c.off;
    return w;
}

}  // namespace

extern "C" {

int64_t fg_scaled_grouped_mm_workspace_bytes(int64_t m_total, int num_groups, int64_t K) {
    if (m_total < 0 || num_groups <= 0 || K <= 0) return -1;
    // The larger of the tables that the call may choose: its N is not known here.  Tables of 256-row blocks hold more
    // padding, those of 128-row blocks more block ids (the larger part above ~32768 rows per group).
    const int64_t single = carve_grouped_mm(nullptr, m_total, num_groups, TILE_ROWS).bytes;
    if (m_total < PAIR_MIN_ROWS * (int64_t)num_groups) return single;
    const int64_t paired = carve_grouped_mm(nullptr, m_total, num_groups, PAIR_ROWS).bytes;
    return single > paired ? single : paired;
}

int fg_scaled_grouped_mm_fp8(void* c, const void* a, const void* b, const float* scale_a, const float* scale_b,
                             const float* bias, int64_t bias_stride_g, const int32_t* offs, int num_groups,
                             int64_t m_total, int64_t N, int64_t K, int64_t ld_a, int64_t ld_c, int out_dtype,
                             void* workspace, int64_t workspace_bytes, void* stream) {
    FG_REQUIRE(m_total >= 0 && N > 0 && K > 0 && num_groups > 0, FG_ERR_INVALID_ARGUMENT, "bad sizes");
    FG_REQUIRE(num_groups <= 1024, FG_ERR_UNSUPPORTED, "at most 1024 groups");
    FG_REQUIRE(K % 16 == 0, FG_ERR_UNSUPPORTED, "K = %lld must be a multiple of 16", (long long)K);
    if (m_total == 0) return FG_OK;
    FG_REQUIRE(c && a && b && scale_a && scale_b && offs && workspace, FG_ERR_INVALID_ARGUMENT, "null pointer");
    FG_REQUIRE((uintptr_t)workspace % 256 == 0, FG_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    FG_REQUIRE(ld_a % 16 == 0 && (uintptr_t)a % 16 == 0, FG_ERR_UNSUPPORTED, "a must have 16-byte aligned rows");
    const bool pairs = use_pairs(m_total, num_groups, N, N);
    const int tile = pairs ? PAIR_ROWS : TILE_ROWS;
    const Workspace ws = carve_grouped_mm(workspace, m_total, num_groups, tile);
    FG_REQUIRE(workspace_bytes >= ws.bytes, FG_ERR_INVALID_ARGUMENT, "workspace holds %lld bytes, needs %lld",
               (long long)workspace_bytes, (long long)ws.bytes);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = fg_group_tiles(offs, num_groups, m_total, tile, ws.sorted_ids, ws.max_pad, ws.expert_ids, ws.n_blocks,
                            ws.post_pad, st);
    if (rc != FG_OK) return rc;
    FgGroupedGemm g{};
    g.sorted_ids = ws.sorted_ids; g.expert_ids = ws.expert_ids; g.num_post_pad = ws.post_pad; g.max_rows = ws.rows;
    g.numel = m_total; g.num_experts = num_groups; g.block_rows = tile; g.cta_pairs = pairs; g.scale_mode = FG_SCALE_VECTOR; g.out_dtype = out_dtype;
    g.c = c; g.a = a; g.w = b; g.a_scale = scale_a; g.w_scale = scale_b; g.bias = bias; g.bias_stride = bias_stride_g;
    // few rows per group: only they are fetched; otherwise a block is one box from its first row
    g.a_rows = m_total; g.gather_div = 1; g.a_contiguous = !use_gather(m_total, num_groups); g.N = N; g.K = K; g.ld_a = ld_a; g.ld_c = ld_c; g.scatter = 1;
    return fg_grouped_gemm(g, st);
}

int64_t fg_moe_routed_workspace_bytes(int64_t n_rows_in, int num_experts, int64_t H, int64_t I) {
    if (n_rows_in < 0 || num_experts <= 0 || H <= 0 || I <= 0) return -1;
    return carve(nullptr, n_rows_in, num_experts, H, I, 2).bytes;
}

int fg_moe_routed_block_fp8_local(void* y, const void* hidden, int hidden_dtype, const void* topk_ids,
                                  int ids_are_i64, const void* topk_w, int topk_w_dtype, int64_t T, int topk,
                                  const void* w1, const void* w2, const float* s1, const float* s2, int num_experts,
                                  int64_t H, int64_t I, void* workspace, int64_t workspace_bytes, void* stream) {
    const int64_t n_in = T * topk;
    int rc = check_dims(n_in, num_experts, H, I, hidden_dtype);
    if (rc != FG_OK) return rc;
    if (n_in == 0) return FG_OK;
    FG_REQUIRE(y && hidden && topk_ids && topk_w && w1 && w2 && s1 && s2 && workspace, FG_ERR_INVALID_ARGUMENT,
               "null pointer");
    FG_REQUIRE((uintptr_t)workspace % 256 == 0, FG_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    const Workspace ws = carve(workspace, n_in, num_experts, H, I, 2);
    FG_REQUIRE(workspace_bytes >= ws.bytes, FG_ERR_INVALID_ARGUMENT, "workspace holds %lld bytes, needs %lld",
               (long long)workspace_bytes, (long long)ws.bytes);
    rc = fg_moe_align(topk_ids, ids_are_i64, n_in, num_experts, TILE_ROWS, nullptr, 0, ws.sorted_ids, ws.max_pad, ws.expert_ids,
                      ws.n_blocks, ws.post_pad, 1, 1, nullptr, nullptr, 0, nullptr, 0, false, (cudaStream_t)stream);
    if (rc != FG_OK) return rc;
    const Experts e{FG_EXPERTS_BLOCK_FP8, hidden, hidden_dtype, topk_w, topk_w_dtype, T, topk, w1, w2, s1, s2, nullptr, nullptr,
                    num_experts, H, I, use_gather(n_in, num_experts), false};
    return run_experts(e, ws, y, (cudaStream_t)stream);
}

int fg_moe_routed_block_fp8_packed(void* y, const void* rows, int64_t R, int64_t row_bytes, const void* w1,
                                   const void* w2, const float* s1, const float* s2, int num_experts, int64_t H,
                                   int64_t I, void* workspace, int64_t workspace_bytes, int out_dtype,
                                   void* const* peer_out, int n_peers, int64_t peer_rows, const int32_t* n_rows_dev,
                                   int64_t region_rows, const int32_t* region_counts, int64_t region_stride,
                                   void* stream) {
    int rc = check_dims(R, num_experts, H, I, out_dtype);
    if (rc != FG_OK) return rc;
    if (R == 0) return FG_OK;
    FG_REQUIRE((y || n_peers > 0) && rows && w1 && w2 && s1 && s2 && workspace, FG_ERR_INVALID_ARGUMENT,
               "null pointer");
    FG_REQUIRE(row_bytes >= H + 4 * (H / 128) + 16 && row_bytes % 16 == 0 && (uintptr_t)rows % 16 == 0,
               FG_ERR_INVALID_ARGUMENT, "bad packed row size %lld", (long long)row_bytes);
    FG_REQUIRE((uintptr_t)workspace % 256 == 0, FG_ERR_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
    const Workspace ws = carve(workspace, R, num_experts, H, I, 2);
    FG_REQUIRE(workspace_bytes >= ws.bytes, FG_ERR_INVALID_ARGUMENT, "workspace holds %lld bytes, needs %lld",
               (long long)workspace_bytes, (long long)ws.bytes);
    const uint8_t* base = reinterpret_cast<const uint8_t*>(rows);
    const int64_t s_cols = H / 128;
    const int32_t* ids = reinterpret_cast<const int32_t*>(base + H + 4 * s_cols);
    const float* wts = reinterpret_cast<const float*>(base + H + 4 * s_cols + 4);
    rc = fg_moe_align_block_size_regions(ids, 0, R, num_experts, TILE_ROWS, nullptr, 0, ws.sorted_ids, ws.max_pad,
                                         ws.expert_ids, ws.n_blocks, ws.post_pad, row_bytes / 4, 1, nullptr,
                                         n_rows_dev, region_rows, region_counts, region_stride, stream);
    if (rc != FG_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    rc = fg_gather_rows_fp8(base, reinterpret_cast<const float*>(base + H), ws.a1, ws.a1s, ws.rows, H, s_cols, row_bytes, row_bytes / 4,
                        ws.sorted_ids, 1, (int32_t)R, ws.post_pad, st);
    if (rc != FG_OK) return rc;
    FgGroupedGemm g{};
    g.sorted_ids = ws.sorted_ids; g.expert_ids = ws.expert_ids; g.num_post_pad = ws.post_pad; g.max_rows = ws.rows;
    g.numel = R; g.num_experts = num_experts; g.block_rows = TILE_ROWS; g.scale_mode = FG_SCALE_BLOCK; g.out_dtype = out_dtype;
    g.c = ws.act; g.a = ws.a1; g.w = w1; g.a_scale = ws.a1s; g.w_scale = s1;
    g.N = 2 * I; g.K = H; g.ld_a = H; g.ld_as = s_cols; g.ld_c = I; g.fuse_silu = 1;
    rc = fg_grouped_gemm(g, st);
    if (rc != FG_OK) return rc;
    rc = fg_quant_rows(FG_QUANT_GROUP128, ws.act, out_dtype, ws.a2, ws.a2s, nullptr, nullptr, ws.rows, I, ws.sorted_ids, 0, (int32_t)R,
                       ws.post_pad, st);
    if (rc != FG_OK) return rc;
    g.c = y; g.a = ws.a2; g.w = w2; g.a_scale = ws.a2s; g.w_scale = s2;
    g.N = H; g.K = I; g.ld_a = I; g.ld_as = I / 128; g.ld_c = H; g.fuse_silu = 0; g.scatter = 1; g.mul_weight = 1;
    g.topk_w = wts; g.topk_w_dtype = FG_DTYPE_F32; g.topk_w_stride = row_bytes / 4;
    if (n_peers > 0) {
        g.dest = reinterpret_cast<const int32_t*>(base + H + 4 * s_cols + 8);
        g.dest_stride = row_bytes / 4;
        g.peer_out = peer_out; g.n_peers = n_peers; g.peer_rows = peer_rows;
    }
    return fg_grouped_gemm(g, st);
}

int fg_moe_routed_block_fp8_local_noalloc(void* y, const void* hidden, int hidden_dtype, const void* topk_ids,
                                          int ids_are_i64, const void* topk_w, int topk_w_dtype, int64_t T,
                                          int topk, const void* w1, const void* w2, const float* s1,
                                          const float* s2, int num_experts, int64_t H, int64_t I, void* stream) {
    int rc = check_dims(T * topk, num_experts, H, I, hidden_dtype);
    if (rc != FG_OK) return rc;
    const int64_t need = carve(nullptr, T * topk, num_experts, H, I, 2).bytes;
    FG_REQUIRE(need <= (int64_t)FG_NOALLOC_SCRATCH_BYTES, FG_ERR_UNSUPPORTED,
               "this problem (T*topk = %lld rows, %d experts, hidden %lld, intermediate %lld) needs %lld bytes of "
               "scratch; the built-in scratch holds %lld. Use fg_moe_routed_block_fp8_local with your own workspace.",
               (long long)(T * topk), num_experts, (long long)H, (long long)I, (long long)need,
               (long long)FG_NOALLOC_SCRATCH_BYTES);
    void* scratch = nullptr;
    rc = builtin_scratch(&scratch);
    if (rc != FG_OK) return rc;
    return fg_moe_routed_block_fp8_local(y, hidden, hidden_dtype, topk_ids, ids_are_i64, topk_w, topk_w_dtype, T, topk,
                                         w1, w2, s1, s2, num_experts, H, I, scratch, FG_NOALLOC_SCRATCH_BYTES, stream);
}

// Workspace of fg_fused_experts in one mode.  num_experts: the larger of the ids' range and the number of weights.
static Workspace carve_experts(void* base, int mode, int64_t T, int topk, int num_experts, int64_t H, int64_t I, int esz) {
    Workspace w{};
    Carver c{reinterpret_cast<uint8_t*>(base), 0};
    const int64_t slots = T * topk;
    const bool pairs = mode != FG_EXPERTS_BLOCK_FP8 && use_pairs(slots, num_experts, 2 * I, H);
    const bool gathered = use_gather(slots, num_experts), plain = mode == FG_EXPERTS_16BIT || mode == FG_EXPERTS_16BIT_SCALED;
    const int64_t cols1 = mode == FG_EXPERTS_BLOCK_FP8 ? H / 128 : 1, cols2 = mode == FG_EXPERTS_BLOCK_FP8 ? I / 128 : 1;
    carve_tables(c, w, slots, num_experts, pairs ? PAIR_ROWS : TILE_ROWS);
    const int64_t rows1 = gathered ? T : w.rows, rows2 = gathered ? slots : w.rows;
    w.scalars = (float*)c.take(4 * (num_experts > 64 ? num_experts : 64));
    w.a1 = c.take(plain ? (gathered ? 0 : rows1 * H * 2) : rows1 * H);
    w.a1s = (float*)c.take(4 * (plain ? w.rows : rows1 * cols1));
    w.act = c.take(rows2 * I * esz);
    w.a2 = c.take(plain ? 0 : rows2 * I);
    w.a2s = (float*)c.take(4 * rows2 * cols2);
    w.routed = c.take(slots * H * esz);
    w.bytes = c.off;
    return w;
}

int64_t fg_fused_experts_workspace_bytes(int mode, int64_t T, int topk, int num_experts, int64_t H, int64_t I,
                                         int hidden_dtype) {
    if (T < 0 || topk <= 0 || num_experts <= 0 || H <= 0 || I <= 0) return -1;
    return carve_experts(nullptr, mode, T, topk, num_experts, H, I, hidden_dtype == FG_DTYPE_F32 ? 4 : 2).bytes;
}

int fg_fused_experts(void* out, const void* hidden, int hidden_dtype, const void* topk_ids, int ids_are_i64, const void* topk_w,
                     int topk_w_dtype, int64_t T, int topk, const void* w1, const void* w2, const float* s1, const float* s2,
                     const float* a1_scale, const float* a2_scale, int mode, int num_experts, int local_experts,
                     const int32_t* expert_map, int expert_map_len, int64_t H, int64_t I, const void* addend, void* workspace,
                     int64_t workspace_bytes, void* stream) {
    FG_REQUIRE(T >= 0 && topk > 0 && num_experts > 0 && local_experts > 0 && H > 0 && I > 0, FG_ERR_INVALID_ARGUMENT, "bad sizes");
    FG_REQUIRE(mode >= FG_EXPERTS_BLOCK_FP8 && mode <= FG_EXPERTS_16BIT_SCALED, FG_ERR_INVALID_ARGUMENT, "bad mode %d", mode);
    if (T == 0) return FG_OK;
    FG_REQUIRE(out && hidden && topk_ids && topk_w && w1 && w2 && workspace && (mode == FG_EXPERTS_16BIT || (s1 && s2)),
               FG_ERR_INVALID_ARGUMENT, "null pointer");
    FG_REQUIRE(T * topk < (1ll << 31), FG_ERR_UNSUPPORTED, "too many route slots");
    // Gathered 16-bit rows are read where they lie; the other orders check their rows when they copy or quantise them.
    FG_REQUIRE(mode < FG_EXPERTS_16BIT || ((uintptr_t)hidden % 16 == 0 && H % 8 == 0), FG_ERR_UNSUPPORTED,
               "hidden rows must be 16-byte aligned (ptr %p, %lld elements)", hidden, (long long)H);
    const int widest = num_experts > local_experts ? num_experts : local_experts;
    const Workspace ws = carve_experts(workspace, mode, T, topk, widest, H, I, hidden_dtype == FG_DTYPE_F32 ? 4 : 2);
    FG_REQUIRE((uintptr_t)workspace % 256 == 0 && workspace_bytes >= ws.bytes, FG_ERR_INVALID_ARGUMENT,
               "workspace holds %lld bytes, needs %lld (256-byte aligned)", (long long)workspace_bytes, (long long)ws.bytes);
    const bool pairs = mode != FG_EXPERTS_BLOCK_FP8 && use_pairs(T * topk, widest, 2 * I, H);
    int rc = fg_moe_align(topk_ids, ids_are_i64, T * topk, num_experts, pairs ? PAIR_ROWS : TILE_ROWS, expert_map, expert_map_len, ws.sorted_ids,
                          ws.max_pad, ws.expert_ids, ws.n_blocks, ws.post_pad, 1, 1, nullptr, nullptr, 0, nullptr, 0, false,
                          (cudaStream_t)stream);
    if (rc != FG_OK) return rc;
    const Experts e{mode, hidden, hidden_dtype, topk_w, topk_w_dtype, T, topk, w1, w2, s1, s2, a1_scale, a2_scale,
                    local_experts, H, I, use_gather(T * topk, widest), pairs};
    rc = run_experts(e, ws, ws.routed, (cudaStream_t)stream);
    if (rc != FG_OK) return rc;
    return fg_moe_sum_indexed(ws.routed, out, T, topk, H, hidden_dtype, nullptr, addend, stream);
}

}  // extern "C"
