// Stands in for libtb200_cuda.so under the native operators: every launcher succeeds without launching anything, the n-th
// product or column sum can be made to fail, all can be made to wait for a word from another thread, and the waits of streams on one another are taken down.
#include "operators.h"

#include <atomic>
#include <chrono>
#include <thread>

typedef cudaStream_t S;

extern "C" {

int fake_fail_at = 0;  // this product or column sum (1: the first one from here on) is refused
int fake_waits = 0;
S fake_log[64][2];
std::atomic<int> fake_closed{0};  // launches return when another thread has set this to 0, or after five seconds with an error

static int wait() {
  const auto until = std::chrono::steady_clock::now() + std::chrono::seconds(5);
  while (fake_closed) {
    if (std::chrono::steady_clock::now() > until) return -78;
    std::this_thread::sleep_for(std::chrono::milliseconds(1));
  }
  return 0;
}
static int launch() { return fake_fail_at > 0 && --fake_fail_at == 0 ? -77 : wait(); }

int tb_gemm_bf16(const void*, const void*, void*, int, int, int, int, int, int, int, int, int, const void*, const void*, void*, int, void*,
                 long long, S) { return launch(); }
int tb_col_sum(const void*, int, int, int, void*, float*, S) { return launch(); }
long long tb_gemm_workspace_bytes(int, int, int) { return 0; }
int tb_stream_wait(S waiter, S signaller) {
  fake_log[fake_waits % 64][0] = waiter;
  fake_log[fake_waits++ % 64][1] = signaller;
  return 0;
}
const char* tb_gemm_last_error() { return ""; }
const char* tb_error_string(int) { return ""; }
const char* tb_last_error() { return ""; }
int tb_layernorm_fwd(const void*, const void*, const void*, void*, float*, float*, int, int, float, S) { return wait(); }
int tb_layernorm_bwd_blocks(int) { return 1; }
int tb_layernorm_bwd_add(const void*, const void*, const void*, const float*, const float*, const void*, void*, void*, void*, float*, int, int, S) { return wait(); }
int tb_attn_fwd(const void*, void*, float*, int, int, int, int, S) { return wait(); }
int tb_attn_bwd(const void*, const void*, const void*, const float*, void*, float*, int, int, int, int, S) { return wait(); }
int tb_embed_fwd(const long long*, const void*, const void*, void*, int, int, int, S) { return wait(); }
int tb_embed_bwd(const long long*, const void*, float*, void*, void*, int, int, int, int, S) { return wait(); }
int tb_xent_fwd(const void*, const long long*, float*, float*, float*, int, int, int, S) { return wait(); }
int tb_xent_bwd(void*, const long long*, const float*, const float*, int, int, int, int, S) { return wait(); }
}
