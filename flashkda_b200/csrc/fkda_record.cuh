// The compact operand record that the forward pass hands from its token-parallel stage to the recurrence, one per (head,
// 32-token chunk), bf16 matrices in core-matrix layout:
//   KN  [32 tok][128 k]   -khat * decay from chunk start (negated: v - k+ S is then one accumulation on top of v)
//   QP  [32 tok][128 k]   qhat * decay from chunk start * scale
//   KR  [32 tok][128 k]   khat * decay to chunk end
//   TB  [32 i][32 j]      T diag(beta),  T = (I + tril(k+ k-^T, -1) diag-row(beta))^-1
//   MQK [32 tok][32 tok]  tril(q+ k-^T)
//   E   [128] fp32        whole-chunk decay per channel
// The recurrence forms U = T diag(beta) (v - k+ S) from v itself.  Against the record of fkda_prepare / fkda_scan (WP, UP
// instead of KN, TB: U = u' - w' S) it is 912 instead of 1104 bytes per token, v is read by the recurrence alone, and the two
// products w', u' with their conversions do not exist; the chain has one more small product per chunk.
#pragma once
#include "fkda_common.cuh"

namespace fkda {
constexpr int kCrKN = 0, kCrQP = 8192, kCrKR = 16384, kCrTB = 24576, kCrMQK = 26624, kCrE = 28672, kCrBytes = 29184;
static_assert(kCrBytes == kCompactRecBytes);
static_assert(kCrBytes <= kRecBytes, "the workspace is sized for the larger record");
}  // namespace fkda
