// The roles of csrc/slot_copies.cuh on host threads: a thread per lane, whole-warp operations that need all 32 lanes, shared-memory
// barriers and a copy engine. bounded_wait.cuh is read as it is (SOURCE: its text without the PTX wrappers' include).
//   sum    the output is the sum of the rows
//   lanes  the launch aborts while half of a summing warp sees its barrier complete and the other half does not yet
//   drain  the launch aborts with copies on their way: none is left when the roles have returned
//   settle an aborting CTA's pause lasts although the sleep in it ends at once
// Exit status 0: right; 2: wrong; 3: a whole-warp operation waits for lanes that have left.
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#define __device__
#define __forceinline__ inline
struct Index { unsigned x; };
static thread_local Index threadIdx;
static Index blockIdx{0};
struct alignas(16) uint4 { uint32_t x, y, z, w; };
struct __nv_bfloat16 { uint16_t bits; };
static float __bfloat162float(__nv_bfloat16 b) { uint32_t u = uint32_t(b.bits) << 16; float f; memcpy(&f, &u, 4); return f; }
static __nv_bfloat16 __float2bfloat16(float f) { uint32_t u; memcpy(&u, &f, 4); return {uint16_t((u + 0x7FFF + ((u >> 16) & 1)) >> 16)}; }
static float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static float __fmul_rn(float a, float b) { return a * b; }
static uint32_t ld_relaxed_gpu(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
static uint32_t ld_acquire_gpu(const uint32_t* p) { return __atomic_load_n(p, __ATOMIC_ACQUIRE); }
static uint32_t atomicExch(uint32_t* p, uint32_t v) { return __atomic_exchange_n(p, v, __ATOMIC_ACQ_REL); }
static uint32_t atomicAdd(uint32_t* p, uint32_t v) { return __atomic_fetch_add(p, v, __ATOMIC_ACQ_REL); }
static uint32_t atomicCAS(uint32_t* p, uint32_t want, uint32_t v) {
  __atomic_compare_exchange_n(p, &want, v, false, __ATOMIC_ACQ_REL, __ATOMIC_ACQUIRE);
  return want;
}
static void __threadfence() {}
static void __syncthreads() {}
static void __nanosleep(unsigned) {}   // may end at once
static uint64_t real_ns() { return std::chrono::steady_clock::now().time_since_epoch().count(); }
static uint64_t globaltimer_ns() { return real_ns() / 5000; }   // so slow that no limit is met by the host's own pace

// ---- warps
struct Warp {
  std::mutex m;
  std::condition_variable cv;
  int here = 0, left = 0;
  uint64_t round = 0;
  uint32_t votes = 0, result = 0;
  std::string op;
};
static thread_local Warp* warp_;
static thread_local unsigned lane_;
static void stuck(const char* op) { printf("%s waits for lanes that have left\n", op); fflush(stdout); _Exit(3); }
static uint32_t meet(const char* op, bool vote) {
  std::unique_lock<std::mutex> l(warp_->m);
  if (warp_->here == 0) { warp_->op = op; warp_->votes = 0; }
  if (warp_->op != op || warp_->left > 0) stuck(op);
  if (vote) warp_->votes |= 1u << lane_;
  const uint64_t round = warp_->round;
  if (++warp_->here == 32) {
    warp_->here = 0;
    warp_->result = warp_->votes;
    ++warp_->round;
    warp_->cv.notify_all();
  } else {
    warp_->cv.wait(l, [&] { return warp_->round != round; });
  }
  return warp_->result;
}
static void leave() {
  std::lock_guard<std::mutex> l(warp_->m);
  ++warp_->left;
  if (warp_->here > 0) stuck(warp_->op.c_str());
}
static void __syncwarp() { meet("__syncwarp", false); }
static bool __all_sync(uint32_t, bool v) { return meet("__all_sync", v) == 0xFFFFFFFFu; }
static bool __any_sync(uint32_t, bool v) { return meet("__any_sync", v) != 0; }

// ---- barriers and the copy engine
struct Bar { int count = 0, pending = 0; long bytes = 0; unsigned phase = 0; };
struct Copy { uint8_t* dst; const void* src; uint32_t bytes; uint64_t* bar; };
static std::mutex g_m;
static std::unordered_map<const uint64_t*, Bar> g_bars;
static std::vector<Copy> g_copies;
static uint8_t* g_smem;
static std::string g_case;
static uint64_t* g_late;          // lanes: the barrier that half of a warp sees complete later
static std::atomic<uint32_t*> g_abort{nullptr};
static std::atomic<uint64_t> g_abort_ns{0};
static void complete(Bar& b) { if (b.pending == 0 && b.bytes == 0) { b.pending = b.count; ++b.phase; } }
static void mbar_init(uint64_t* bar, uint32_t n) { std::lock_guard<std::mutex> l(g_m); g_bars[bar] = Bar{int(n), int(n), 0, 0}; }
static void mbar_arrive(uint64_t* bar) { std::lock_guard<std::mutex> l(g_m); Bar& b = g_bars[bar]; --b.pending; complete(b); }
static void mbar_arrive_expect_tx(uint64_t* bar, uint32_t n) {
  std::lock_guard<std::mutex> l(g_m);
  Bar& b = g_bars[bar];
  b.bytes += n;
  --b.pending;
  complete(b);
}
static void raise_abort() {
  uint64_t none = 0;
  if (g_abort_ns.compare_exchange_strong(none, real_ns())) atomicExch(g_abort.load(), 1u);
}
static bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  bool done;
  unsigned phase;
  {
    std::lock_guard<std::mutex> l(g_m);
    phase = g_bars[bar].phase;
    done = (phase & 1u) != parity;
  }
  if (!done) std::this_thread::sleep_for(std::chrono::microseconds(50));
  if (bar == g_late && threadIdx.x / 32 == 6 && lane_ < 16 && phase >= 2) { raise_abort(); return false; }
  return done;
}
static uint32_t smem_u32(const void* p) { return uint32_t(static_cast<const uint8_t*>(p) - g_smem); }
static void bulk_load(uint32_t dst, const void* src, uint32_t n, uint64_t* bar) {
  std::lock_guard<std::mutex> l(g_m);
  g_copies.push_back({g_smem + dst, src, n, bar});
}
static void fence_proxy_async() {}

#include SOURCE
#include "slot_copies.cuh"

using namespace mono;
constexpr int H = 512, SLOTS = 8, TILE = 128, ITEMS = 21, T = kGrid * ITEMS - 5;
struct Params {
  int num_tokens = T, sh_on = 1, sh_part = 1, sh_parts = 3;
  const __nv_bfloat16* partial;
  const __nv_bfloat16* residual;
  __nv_bfloat16* out;
  float out_scale = 0.5f;
};
static __nv_bfloat16 value(size_t row, int col, int salt) { return __float2bfloat16(float((row * 37 + size_t(col) * 11 + salt) % 255) - 127.f); }

int main(int, char** argv) {
  g_case = argv[1];
  if (g_case == "settle") {
    const uint64_t t0 = globaltimer_ns();
    settle();
    return globaltimer_ns() - t0 >= 200000 ? 0 : 2;
  }
  const uint32_t first = 77;
  std::vector<__nv_bfloat16> partial(size_t(T) * (SLOTS + 1) * H), residual(size_t(T) * H), out(size_t(T) * H);
  for (uint32_t tok = first; tok < T; tok += kGrid)
    for (int c = 0; c < H; ++c) {
      for (int k = 0; k < SLOTS; ++k) partial[(size_t(tok) * SLOTS + k) * H + c] = value(size_t(tok) * SLOTS + k, c, 1);
      partial[(size_t(T) * SLOTS + tok) * H + c] = value(tok, c, 2);
      residual[size_t(tok) * H + c] = value(tok, c, 3);
    }
  Params p;
  p.partial = partial.data();
  p.residual = residual.data();
  p.out = out.data();
  constexpr uint32_t SMEM = 5 * (SLOTS + 2) * H * 2 + 100;
  std::vector<uint4> smem(SMEM / 16 + 1);
  g_smem = reinterpret_cast<uint8_t*>(smem.data());
  SumBars bars;
  for (int s = 0; s < kSumStages; ++s) { mbar_init(&bars.full[s], 1); mbar_init(&bars.empty[s], kSumWarps); }
  static Workspace ws;
  g_abort = &ws.abort_flag;
  const WaitCtx wc{&ws, ~0ull};
  if (g_case == "lanes") g_late = &bars.full[1];

  std::atomic<bool> stop{false};
  std::thread engine([&] {
    size_t landed = 0;
    while (!stop) {
      Copy c{};
      {
        std::lock_guard<std::mutex> l(g_m);
        // drain: what the third round of the stages asks for lands a while after the abort
        const bool held = g_case == "drain" && landed >= 100 && (g_abort_ns == 0 || real_ns() - g_abort_ns < 400000000);
        if (held && g_copies.size() >= 30) raise_abort();
        if (!held && !g_copies.empty()) { c = g_copies.back(); g_copies.pop_back(); }
      }
      if (c.dst == nullptr) { std::this_thread::sleep_for(std::chrono::microseconds(20)); continue; }
      memcpy(c.dst, c.src, c.bytes);
      ++landed;
      std::lock_guard<std::mutex> l(g_m);
      Bar& b = g_bars[c.bar];
      b.bytes -= c.bytes;
      complete(b);
    }
  });
  constexpr int WARPS = 12;
  std::vector<Warp> warps(WARPS);
  std::vector<std::thread> lanes;
  for (int t = 0; t < WARPS * 32; ++t)
    lanes.emplace_back([&, t] {
      threadIdx.x = t;
      warp_ = &warps[t / 32];
      lane_ = t % 32;
      SlotCopies<H, SLOTS, TILE, Params> copies(p, bars, wc, g_smem, SMEM);
      if (t / 32 == 0) copies.request(first, lane_);
      else if (t / 32 >= WARPS - kSumWarps) copies.add(first, t - (WARPS - kSumWarps) * 32, lane_);
      leave();
    });
  for (auto& l : lanes) l.join();
  size_t on_their_way;
  { std::lock_guard<std::mutex> l(g_m); on_their_way = g_copies.size(); }
  stop = true;
  engine.join();
  if (on_their_way != 0) { printf("%zu copies on their way\n", on_their_way); return 2; }
  if (g_case != "sum") return ws.abort_flag != 0 ? 0 : 2;
  for (uint32_t tok = first; tok < T; tok += kGrid)
    for (int c = 0; c < H; ++c) {
      float s = 0.f, base = 0.f;
      for (int k = 0; k < SLOTS; ++k) s += __bfloat162float(value(size_t(tok) * SLOTS + k, c, 1));
      if (int(tok / TILE) % p.sh_parts == p.sh_part) base += __bfloat162float(value(tok, c, 2));
      base += __bfloat162float(value(tok, c, 3));
      if (out[size_t(tok) * H + c].bits != __float2bfloat16(s * p.out_scale + base).bits) { printf("token %u column %d\n", tok, c); return 2; }
    }
  return ws.abort_flag == 0 ? 0 : 2;
}
