// Downloads when the system has no pinned memory left, and when a conversion
// cannot be launched: the library's own pinned allocation (bf::host_alloc) is
// replaced by one that fails on request.
//   stage_model pinned   every download still arrives, through another way
//   stage_model drain    a download that fails returns with its stream idle
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "../code_mojo_gb300/csrc/bf_internal.h"

static bool g_none_left = false;
static int g_refused = 0;

namespace bf {
void* host_alloc(size_t bytes) {
  if (g_none_left) {
    ++g_refused;
    throw Error{BF_ENOMEM, "no pinned memory left"};
  }
  void* p = nullptr;
  if (cudaHostAlloc(&p, bytes < 64 ? 64 : bytes, cudaHostAllocDefault) != cudaSuccess) throw Error{BF_ENOMEM, "cudaHostAlloc"};
  return p;
}
}  // namespace bf

using namespace bf;

static int check(const char* what, const std::vector<double>& got, const std::vector<double>& want) {
  if (std::memcmp(got.data(), want.data(), want.size() * sizeof(double)) == 0) return 0;
  std::printf("%s differs\n", what);
  return 1;
}

static int pinned() {
  int bad = 0;
  for (int n : {5, 13, 18, 20}) {
    for (int dtype : {BF_C128, BF_C64}) {
      const size_t N = (size_t)1 << n;
      std::vector<double> re(N), im(N);
      for (size_t i = 0; i < N; ++i) {
        re[i] = (double)(float)(1.0 + 0.001 * (double)i);
        im[i] = -(double)(float)(0.5 * (double)i);
      }
      bf_state* st = nullptr;
      if (bf_state_create(n, dtype, &st) != BF_OK) return 10;
      if (bf_state_upload_soa(st, re.data(), im.data()) != BF_OK) return 11;
      g_none_left = true;
      g_refused = 0;
      std::vector<double> r(N, 7.0), i(N, 7.0);
      const int rc = bf_state_download_soa(st, r.data(), i.data());
      g_none_left = false;
      if (rc != BF_OK) {
        std::printf("state of %d qubits, dtype %d: error %d\n", n, dtype, rc);
        ++bad;
      } else {
        bad += check("re", r, re) + check("im", i, im);
      }
      bf_state_destroy(st);
    }
  }
  // a batch of two circuits: X on qubit 0
  for (int dtype : {BF_C128, BF_C64}) {
    bf_op op;
    std::memset(&op, 0, sizeof op);
    op.kind = BF_OP_GATE;
    op.gate = BF_GATE_X;
    const bf_op* lists[2] = {&op, &op};
    const int32_t nq[2] = {3, 14};
    const int64_t nops[2] = {1, 1};
    bf_batch* b = nullptr;
    if (bf_batch_create(2, nq, lists, nops, dtype, nullptr, &b) != BF_OK) return 12;
    if (bf_batch_run(b, 1) != BF_OK) return 13;
    for (int c = 0; c < 2; ++c) {
      std::vector<double> r((size_t)1 << nq[c], 7.0), i(r), er(r.size(), 0.0), ei(r.size(), 0.0);
      er[1] = 1.0;
      g_none_left = true;
      const int rc = bf_batch_download(b, c, r.data(), i.data());
      g_none_left = false;
      if (rc != BF_OK) {
        std::printf("batch, dtype %d: error %d\n", dtype, rc);
        ++bad;
      } else {
        bad += check("batch re", r, er) + check("batch im", i, ei);
      }
    }
    bf_batch_destroy(b);
  }
  if (g_refused == 0) {
    std::printf("no allocation was refused: the replacement did not take\n");
    ++bad;
  }
  return bad ? 1 : 0;
}

// The second chunk's conversion fails while the stream is busy with the first.
static int drain() {
  cudaStream_t s;
  void* d = nullptr;
  const size_t big = (size_t)1 << 30;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess || cudaMalloc(&d, big) != cudaSuccess) return 20;
  const uint64_t count = 2 * kHostChunk;
  std::vector<double> re(count), im(count);
  HostStage stage;
  if (!stage.reserve(count)) return 21;
  int chunk = 0, rc = 0;
  bool failed = false;
  try {
    stage.download(count, re.data(), im.data(), s, [&](double*, double*, uint64_t, uint64_t) {
      if (chunk++ == 1) throw Error{BF_ECUDA, "no launch"};
      for (int k = 0; k < 40; ++k) cudaMemsetAsync(d, k, big, s);  // several milliseconds
    });
  } catch (const Error&) {
    failed = true;
    if (cudaStreamQuery(s) != cudaSuccess) {
      std::printf("the download returned with its stream busy\n");
      rc = 1;
    }
  }
  cudaStreamSynchronize(s);
  stage.release();
  cudaFree(d);
  cudaStreamDestroy(s);
  return failed ? rc : 22;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "pinned")) return pinned();
  if (argc == 2 && !std::strcmp(argv[1], "drain")) return drain();
  return 2;
}
