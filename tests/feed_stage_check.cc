// FeedStage on the host alone: the CUDA calls it makes are stood in for here, and copies run only when their stream is
// synchronised, so data that are overwritten while a flushed batch still reads them show up as wrong bytes. Built with
// AddressSanitizer, which watches the ends of the staging buffer.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "feed_stage.h"

struct Launch { const xb_copy_item* items; int n; cudaStream_t stream; };
static std::vector<Launch> g_queue;
static int g_flushes = 0;

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
const char* xb_last_error(void) { return ""; }
int xb_copy_segments(const xb_copy_item* items, int32_t n, int64_t max_bytes, xb_stream_t stream) {
  for (int i = 0; i < n; ++i)
    if (items[i].bytes > max_bytes) abort();
  g_queue.push_back(Launch{items, n, (cudaStream_t)stream});
  ++g_flushes;
  return 0;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::vector<Launch> later;
  for (const Launch& l : g_queue) {
    if (l.stream != s) { later.push_back(l); continue; }
    for (int i = 0; i < l.n; ++i) memcpy(l.items[i].dst, l.items[i].src, (size_t)l.items[i].bytes);
  }
  g_queue = later;
  return cudaSuccess;
}
}

struct TestBlob {
  std::vector<unsigned char> device, want;
  template <typename T> T* as() { return reinterpret_cast<T*>(device.data()); }
};
typedef blaze::FeedStage<TestBlob> Stage;
static const cudaStream_t S1 = (cudaStream_t)1, S2 = (cudaStream_t)2;

static void Feed(Stage& st, TestBlob& b, size_t len, unsigned seed, cudaStream_t s) {
  std::vector<unsigned char> data(len);
  for (size_t i = 0; i < len; ++i) data[i] = (unsigned char)(seed * 131 + i * 7 + (i >> 8));
  if (b.device.size() < len) {                                  // grows as a blob does: after what writes it has run
    if (st.pending(&b)) st.Flush(s);
    cudaStreamSynchronize(S1); cudaStreamSynchronize(S2);
    b.device.resize(len, 0xEE);
  }
  st.Add(&b, data.data(), len, s);
  b.want = data;                                                // `data` goes away: the caller's buffer is free after Add
}
static void Finish(Stage& st, cudaStream_t s) { st.Flush(s); cudaStreamSynchronize(s); st.Done(); }
static void Check(const char* what, const TestBlob& b) {
  if (memcmp(b.device.data(), b.want.data(), b.want.size()) != 0) { fprintf(stderr, "%s: wrong bytes\n", what); exit(1); }
}

int main() {
  {  // one input fed again and again before anything reads it
    for (size_t len : {(size_t)1, (size_t)1000, Stage::kMaxFeed}) {
      Stage st;
      TestBlob b;
      for (unsigned i = 0; i < 2000; ++i) Feed(st, b, len, i, S1);
      Finish(st, S1);
      Check("same length again", b);
    }
    Stage st;
    TestBlob b;
    for (unsigned i = 0; i < 2000; ++i) Feed(st, b, Stage::kMaxFeed - i % 3, i, S1);
    Finish(st, S1);
    Check("other lengths", b);
    TestBlob c;
    for (unsigned i = 0; i < 2000; ++i) { Feed(st, c, 5000, i, S1); st.Drop(&c); }      // replaced by what goes another way
    if (st.pending(&c)) { fprintf(stderr, "dropped feed waits\n"); return 1; }
    Feed(st, c, 5000, 7, S1);
    Finish(st, S1);
    Check("fed after drops", c);
  }
  {  // more inputs than descriptors, more bytes than the buffer
    for (size_t len : {(size_t)16, Stage::kMaxFeed}) {
      Stage st;
      std::vector<TestBlob> b(Stage::kMaxItems * 2 + 3);
      for (int pass = 0; pass < 3; ++pass) {
        for (size_t i = 0; i < b.size(); ++i) Feed(st, b[i], len, (unsigned)(i + pass), S1);
        Finish(st, S1);
        for (TestBlob& x : b) Check("many", x);
      }
    }
  }
  {  // a batch enqueued on one stream is waited for before its arrays are overwritten from another
    Stage st;
    TestBlob a, b;
    Feed(st, a, 3000, 1, S1);
    st.Flush(S1);
    const std::vector<unsigned char> first = a.want;
    Feed(st, b, 3000, 2, S2);
    Finish(st, S2);
    if (memcmp(a.device.data(), first.data(), first.size()) != 0) { fprintf(stderr, "in flight: overwritten\n"); return 1; }
    Check("second stream", b);
  }
  // any order of feeds, drops and flushes: what was fed last arrives
  std::mt19937 rng(1);
  for (int trial = 0; trial < 200; ++trial) {
    Stage st;
    std::vector<TestBlob> b(1 + rng() % 200);
    std::vector<bool> fed(b.size(), false);
    for (int step = 0; step < 400; ++step) {
      const size_t i = rng() % b.size();
      switch (rng() % 8) {
        case 0: st.Flush(S1); break;
        case 1: st.Drop(&b[i]); b[i].want.clear(); break;       // (whatever the blob holds then)
        default: Feed(st, b[i], 1 + rng() % (rng() % 4 ? 2000 : Stage::kMaxFeed), rng(), S1);
      }
    }
    Finish(st, S1);
    for (TestBlob& x : b) Check("random", x);
  }
  printf("ok %d\n", g_flushes);
  return 0;
}
