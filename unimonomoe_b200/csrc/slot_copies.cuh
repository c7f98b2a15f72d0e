// The slot sum where the copy engine brings a token's partial rows through shared memory (FORM_COPIES): one warp of a CTA requests
// them, kSumWarps others add them. Rows are in slot order and a token's rows neighbours; one row to a slot.
#pragma once
#include "bounded_wait.cuh"

namespace mono {

constexpr int kSumStages = 8;   // at most; a stage holds the rows of one token
constexpr int kSumWarps = 8;

struct SumBars {
  uint64_t full[kSumStages], empty[kSumStages];   // empty: one arrival per summing warp
};

// P: num_tokens, partial, out, out_scale, residual, sh_on, sh_part, sh_parts (the kernel's parameters). H columns; tokens are dealt to
// the shared expert's ranks in tiles of TILE.
template <int H, int SLOTS, int TILE, class P>
struct SlotCopies {
  static constexpr int W = 8;                // bf16 per 16-byte vector
  static constexpr uint32_t ROW_BYTES = H * 2;

  const P& p;
  SumBars& bars;
  const WaitCtx& wc;
  uint8_t* buf;            // shared memory of the stages
  uint32_t stages, stage_bytes;

  __device__ __forceinline__ SlotCopies(const P& params, SumBars& barriers, const WaitCtx& ctx, uint8_t* smem, uint32_t smem_bytes)
      : p(params), bars(barriers), wc(ctx), buf(smem) {
    stage_bytes = (SLOTS + (p.sh_on ? 1 : 0) + (p.residual != nullptr ? 1 : 0)) * ROW_BYTES;
    stages = smem_bytes / stage_bytes;
    if (stages > kSumStages) stages = kSumStages;
  }
  __device__ __forceinline__ bool shared_row(uint32_t tok) const {   // this launch computed the shared expert for the token
    return p.sh_on && static_cast<int>(tok / TILE) % p.sh_parts == p.sh_part;
  }

  // One warp: rows of tokens first, first + kGrid, ... until the launch aborts. Behind it all of them have come in.
  __device__ __forceinline__ void request(uint32_t first, int lane) const {
    static_assert(SLOTS <= 32, "a lane requests one row");
    const uint32_t tokens = static_cast<uint32_t>(p.num_tokens), buf_u32 = smem_u32(buf);
    // the rows were written by other SMs, some by ordinary stores; the copies read them through the async proxy
    fence_proxy_async();
    uint32_t n = 0;
    for (uint32_t tok = first; tok < tokens; tok += kGrid, ++n) {
      const uint32_t st = n % stages;
      const bool sh = shared_row(tok);
      if (!mbar_wait_warp(&bars.empty[st], ((n / stages) & 1u) ^ 1u, wc, kSiteSumEmpty)) break;
      if (lane == 0) mbar_arrive_expect_tx(&bars.full[st], (SLOTS + (sh ? 1 : 0) + (p.residual != nullptr ? 1 : 0)) * ROW_BYTES);
      __syncwarp();
      const uint32_t dst = buf_u32 + st * stage_bytes;
      if (lane < SLOTS)   // a row each
        bulk_load(dst + lane * ROW_BYTES, p.partial + (static_cast<size_t>(tok) * SLOTS + lane) * H, ROW_BYTES, &bars.full[st]);
      if (sh && lane == 0)
        bulk_load(dst + SLOTS * ROW_BYTES, p.partial + (static_cast<size_t>(tokens) * SLOTS + tok) * H, ROW_BYTES, &bars.full[st]);
      if (p.residual != nullptr && lane == 0)
        bulk_load(dst + (SLOTS + (p.sh_on ? 1 : 0)) * ROW_BYTES, p.residual + static_cast<size_t>(tok) * H, ROW_BYTES, &bars.full[st]);
    }
    drain_copies(bars.full, n, stages);
  }

  // kSumWarps warps, thread v of them: vector v of the same tokens, until the launch aborts.
  __device__ __forceinline__ void add(uint32_t first, int v, int lane) const {
    static_assert(H / W <= kSumWarps * 32, "a thread has one vector of a row");
    const uint32_t tokens = static_cast<uint32_t>(p.num_tokens);
    uint32_t n = 0;
    for (uint32_t tok = first; tok < tokens; tok += kGrid, ++n) {
      const uint32_t st = n % stages;
      // the whole warp waits and gives up as one: lanes that left alone would be missed at the __syncwarp below
      if (!mbar_wait_warp(&bars.full[st], (n / stages) & 1u, wc, kSiteSumFull)) return;
      if (v < H / W) {
        const uint8_t* src = buf + st * stage_bytes + v * 16;
        float s[W], base[W];
#pragma unroll
        for (int i = 0; i < W; ++i) s[i] = base[i] = 0.f;
        auto add_row = [&](float (&d)[W], int r) {
          const uint4 raw = *reinterpret_cast<const uint4*>(src + r * ROW_BYTES);
          const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
          for (int i = 0; i < W; ++i) d[i] += __bfloat162float(b[i]);
        };
#pragma unroll
        for (int r = 0; r < SLOTS; ++r) add_row(s, r);
        if (shared_row(tok)) add_row(base, SLOTS);
        if (p.residual != nullptr) add_row(base, SLOTS + (p.sh_on ? 1 : 0));
        __nv_bfloat16 o[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
          o[i] = __float2bfloat16(p.sh_on || p.residual != nullptr ? __fmaf_rn(s[i], p.out_scale, base[i]) : __fmul_rn(s[i], p.out_scale));
        *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(tok) * H + v * W) = *reinterpret_cast<const uint4*>(o);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.empty[st]);
    }
  }
};

}  // namespace mono
