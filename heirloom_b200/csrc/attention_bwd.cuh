// What the two attention backward kernels (heads of 64 and of 128 channels) share.
#pragma once
#include <type_traits>

#include "kernels.h"

namespace hl {

struct FbParams {
  int B, T, H;
  const float* lse;    // [B,H,T]
  const float* delta;  // [B,H,T] rowsum(dO * O)
  float scale, scale_log2;
  int* status;
};

// Heads of 128 channels.  Keys as rows (attention_bwd_t.cu): boxes of 64 channels by 128 rows by one batch entry in mq, mk, mv and mdo, of 32 f32 channels by
// 32 rows in mdq, of 64 channels by 32 keys in mdk and mdv.
int launch_attention_bwd_t(hl_ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                           const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const FbParams& p);
// Queries as rows (attention_bwd128.cu): key tiles of 64 rows in mk and mv, query tiles of 128 in mq and mdo; the rest as for the 64-channel kernel.
int launch_attention_bwd128(hl_ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo,
                            const CUtensorMap& mdq, const CUtensorMap& mdk, const CUtensorMap& mdv, const FbParams& p);

}  // namespace hl
