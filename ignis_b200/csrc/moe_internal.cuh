// Types shared by the MoE entry points and grouping (moe.cu) and the kernels behind them.
#ifndef B200Q_MOE_INTERNAL_CUH
#define B200Q_MOE_INTERNAL_CUH

#include "../../include/ignis_moe.h"

#include "common.cuh"

namespace b200q {

constexpr uint32_t kStatusBadExpert = 1u, kStatusAbsentRecord = 2u, kStatusRange = 4u;
constexpr uint32_t kStatusTcWait = 8u;   // a bounded wait of the tensor-core expert kernels ran out

// A work item: up to kMoeTcItemRows sorted rows of one expert.
struct Item {
  uint32_t expert, first, count, pad;
};

struct ExpertParams {
  const int32_t *ids;        // expert of every assignment: [tokens][top_k]
  const ignis_moe_slot *slots;
  const Item *items;
  const uint32_t *n_items;  // items
  const uint32_t *sorted;   // row -> assignment index (token * top_k + rank)
  const uint16_t *x;        // BF16 [tokens][hidden]
  const float *weights;     // routing weights [tokens][top_k]
  uint16_t *x_rows;         // rotated x: fp16 [rows][hidden]
  float *x_scale;           // inverse scale per row
  float *gu;                // fp32 [rows][2 inter]: gate | up products
  uint16_t *h_rows;         // rotated silu(g) u: fp16 [rows][inter]
  float *h_scale;
  float *down_rows;         // fp32 [tokens][top_k][hidden]: the weighted down products, before they are added
  long long *acc;           // int64 [tokens][hidden]
  uint32_t *status;
  uint32_t hidden, inter, top_k, experts;
};


// The routed experts on the tensor cores (moe_tc.cu): rows rotated once into fp16 rows with one
// scale per row, items multiplied with their expert's records by tcgen05.
int32_t moe_tc_prepare(ErrorSlot &slot);
constexpr uint32_t kMoeTcItemRows = 192;
constexpr uint32_t kMoeNarrowTokens = 64;   // calls of up to this many tokens may share an accumulator with others at work
int32_t moe_tc_experts(ErrorSlot &slot, const DeviceState &dev, const ExpertParams &p, uint32_t rows, uint32_t items_max,
                       const uint32_t *offsets, cudaStream_t stream, const char *what);

// The shared expert of a wide call on the tensor cores (moe_fp8_tc.cu): FP8 rows widened exactly to
// BF16 in swizzled shared memory, BF16 activations by TMA, tcgen05 kind::f16. Takes calls of more
// than 64 tokens, by the work they are (moe_fp8_tc.cu), whose widths are multiples of 128 and whose x and h are
// 16-byte aligned.
int32_t moe_fp8_tc_prepare(ErrorSlot &slot);
bool moe_fp8_tc_takes(const DeviceState &dev, uint32_t hidden, uint32_t inter, uint32_t tokens, const void *x, const void *h);
cudaError_t moe_fp8_tc_shared_expert(const DeviceState &dev, const uint8_t *gate, const uint8_t *up, const uint8_t *down, const uint16_t *x,
                                     uint32_t tokens, uint32_t hidden, uint32_t inter, void *h, float *shared, cudaStream_t stream);
cudaError_t moe_fp8_tc_status(uint32_t *status, cudaStream_t stream);   // non-zero: one of its bounded waits ran out

// The narrow dense products of the block (moe_rows.cu): the router's logits and selection, and the
// shared expert of calls the tensor-core kernels do not take.
int32_t moe_rows_prepare(ErrorSlot &slot);
cudaError_t moe_router_logits_launch(const DeviceState &dev, const uint16_t *x, const uint16_t *w, uint32_t tokens, uint32_t hidden,
                                     uint32_t experts, float *logits, cudaStream_t stream);
cudaError_t moe_router_select_launch(const DeviceState &dev, const float *logits, uint32_t tokens, uint32_t experts, uint32_t top_k,
                                     int32_t *ids, float *weights, cudaStream_t stream);
cudaError_t moe_rows_shared_expert(const DeviceState &dev, const uint8_t *gate, const uint8_t *up, const uint8_t *down, const uint16_t *x,
                                   uint32_t tokens, uint32_t hidden, uint32_t inter, void *h, float *shared, cudaStream_t stream);

}  // namespace b200q

#endif
