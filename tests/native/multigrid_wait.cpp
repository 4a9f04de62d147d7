// A multigrid solve whose waits run out, and the solves after it (run by test_multigrid_wait_gpu.py). The wait
// across the grid is cut to one poll, which the block that arrives first cannot pass: every block still runs
// to the end, on values that nothing ordered.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "amg.hpp"

using namespace rsg;

namespace {

// five-point Laplacian of an m x m grid plus a small diagonal
Csr laplacian(int m) {
  Csr A;
  A.n = A.m = m * m;
  A.ptr.push_back(0);
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) {
      auto add = [&](int a, int b, double v) {
        if (a >= 0 && a < m && b >= 0 && b < m) A.col.push_back(a * m + b), A.val.push_back(v);
      };
      add(i - 1, j, -1.0), add(i, j - 1, -1.0), add(i, j, 4.001), add(i, j + 1, -1.0), add(i + 1, j, -1.0);
      A.ptr.push_back((int)A.col.size());
    }
  return A;
}

void need(bool ok, const char *what) {
  if (!ok) std::printf("failed: %s\n", what), std::exit(1);
}

int report(AmgDevice &D) {  // the status check() raises
  try {
    D.check();
  } catch (const Error &e) {
    return e.code;
  }
  return RS_OK;
}

}  // namespace

int main() {
  rs_ctx *ctx = nullptr;
  need(rs_ctx_create(0, &ctx) == RS_OK, "context");
  {
    const Csr A = laplacian(90);
    const size_t n = (size_t)A.n;
    AmgDevice D;
    D.upload(amg_setup(A), ctx->stream);
    const unsigned polls = D.wait_polls;
    for (int C : {6, 9, 12}) {
      std::vector<float> b(n * C), want(n * C), got(n * C);
      for (size_t i = 0; i < b.size(); ++i) b[i] = std::sin(0.37f * (float)i);
      DevBuf<float> bd(b.size()), xd(b.size());
      auto solve = [&](std::vector<float> &out) {
        D.pcg(ctx, bd.p, xd.p, C, 3);
        xd.download(out.data(), out.size(), ctx->stream);
        RSG_CUDA("test", cudaStreamSynchronize(ctx->stream));
      };
      bd.upload(b.data(), b.size(), ctx->stream);
      solve(want);
      need(report(D) == RS_OK, "a solve reports nothing");
      // seen when the stream has been waited for, once
      D.wait_polls = 1;
      solve(got);
      need(report(D) == RS_GPU, "a wait that runs out is reported");
      need(report(D) == RS_OK, "it is reported once");
      // seen by the next solve when nobody asked
      solve(got);
      D.wait_polls = polls;
      int code = RS_OK;
      try {
        solve(got);
      } catch (const Error &e) {
        code = e.code;
      }
      need(code == RS_GPU, "the next solve reports it");
      // and the solves after it are what they were
      for (int k = 0; k < 2; ++k) {
        solve(got);
        need(report(D) == RS_OK, "the solve after it reports nothing");
        need(got == want, "the solve after it gives the same bits");
      }
    }
  }
  rs_ctx_free(ctx);
  std::printf("ok\n");
  return 0;
}
