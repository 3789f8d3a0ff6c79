// CPU replay of gathered plans (test driver): the plan build_plan makes with
// gather = true, replayed as the tensor-core kernel consumes it, against the
// plain plan of the same matrix.
//   * every nonzero is in exactly one block, gathered or kept, of its row;
//   * a gathered block and its B tile name the same rows of B;
//   * C in FP64 equals the CSR product;
//   * with infinite and NaN values in B, C holds the same NaNs and infinities
//     as the plain plan's (stored zeros times such a value are NaN).
// Prints "ALL OK" or "FAIL"; exit status 0 on success.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "smat_internal.h"

namespace smat {
void set_error(const std::string& m) { std::fprintf(stderr, "error: %s\n", m.c_str()); }
smat_status fail(smat_status st, const std::string& m) {
  set_error(m);
  return st;
}
}  // namespace smat

using namespace smat;

namespace {

int bad = 0;
void check(bool ok, const char* what) {
  if (!ok && bad++ < 20) std::printf("  violated: %s\n", what);
}

// C of a plan, as the kernel and its epilogue make it.
std::vector<double> replay(const HostBcsr& hb, const Plan& pl, int R, int cls, const std::vector<double>& B, int N,
                           std::vector<int>* seen) {
  const int bh = hb.bh, PW = R % kMmaWarps == 0 ? R / kMmaWarps : 0;
  std::vector<double> C((size_t)hb.rows_p * N, 0.0);
  bool any_odd = false;
  for (double x : B) any_odd |= !std::isfinite(x);
  for (int p = 0; p < pl.n_panels; p++) {
    const PanelInfo& pi = pl.panels[p];
    std::vector<double> acc((size_t)R * bh * N, 0.0);
    for (int c = 0; c < pi.nstages; c++) {
      const StageRec& st = pl.stages[pi.stage_off + c];
      check(st.nblk <= stage_rows(cls) / bh && st.ntiles <= stage_tiles(cls), "stage size");
      check(stage_hdr_max(st.nblk) <= kStageHdrBytes, "header size");
      const uint8_t* h = pl.headers.data() + st.hdr_off;
      uint16_t wl[kMmaWarps];
      std::memcpy(wl, h, sizeof(wl));
      uint32_t gmask;
      std::memcpy(&gmask, h + 12, 4);
      // gathered tiles last, their lists of rows one after the other
      const int na = st.ntiles - st.ngath;
      for (int t = 0; t < st.ntiles; t++)
        check(t < na ? st.kb[t] >= 0 : st.kb[t] == st.kb[na] - (t - na), "gathered tiles last and consecutive");
      int covered = 0;
      for (int w = 0; w < kMmaWarps; w++)
        for (int e = 0; e < (wl[w] >> 8); e++) {
          uint32_t m;
          std::memcpy(&m, h + kStageHdrFixed + 4 * ((wl[w] & 0xff) + e), 4);
          const int pos = m & 31, tile = (m >> 5) & 15, slot = (m >> 9) & 31, len = ((m >> 14) & 15) + 1;
          const bool accumulate = (m >> 18) & 1;
          check(slot * kMmaWarps / R == w && (slot + len - 1) * kMmaWarps / R == w, "slot owner");
          for (int q = 0; q < len; q++) {
            covered++;
            const int32_t blk = pl.stream_blk[st.blk_off + pos + q];
            check((blk < 0) == (((gmask >> (pos + q)) & 1u) != 0), "gathered mask");
            int64_t src[16];
            int64_t rows[16];
            for (int j = 0; j < 16; j++) {
              if (blk < 0) {
                check(st.kb[tile] == blk && len == 1, "a gathered block has its own tile");
                src[j] = pl.gsrc[(size_t)(-(blk + 1)) * 16 + j];
                rows[j] = pl.gcol[(size_t)(-(blk + 1)) * 16 + j];
                if (src[j] >= 0) check(hb.colidx[src[j] / 16] + src[j] % 16 == rows[j], "row of B");
              } else {
                check(st.kb[tile] * 16 == hb.colidx[blk], "tile of a kept block");
                src[j] = (int64_t)blk * 16 + j;
                rows[j] = hb.colidx[blk] + j;
              }
              if (src[j] >= 0 && seen) (*seen)[src[j]]++;
            }
            const int sl = slot + q;
            for (int i = 0; i < bh; i++)
              for (int n = 0; n < N; n++) {
                double s = 0;
                for (int j = 0; j < 16; j++) {
                  const double a = src[j] < 0 ? 0.0 : hb.val[(src[j] / 16) * bh * 16 + i * 16 + src[j] % 16];
                  s += a * (rows[j] < 0 ? 0.0 : B[(size_t)rows[j] * N + n]);
                }
                double& d = acc[((size_t)sl * bh + i) * N + n];
                d = accumulate ? d + s : s;
              }
          }
        }
      check(covered == st.nblk, "every block of the stage in one entry");
    }
    for (int s = 0; s < R; s++) {
      if ((pi.ext_mask >> s) & 1u) continue;
      std::vector<uint8_t> nan(N, 0);
      if (any_odd && !pl.poison_ptr.empty())
        for (int32_t q = pl.poison_ptr[(size_t)p * R + s]; q < pl.poison_ptr[(size_t)p * R + s + 1]; q++)
          for (int c = 0; c < 16; c++)
            if ((pl.poison[q].mask >> c) & 1)
              for (int n = 0; n < N; n++) nan[n] |= !std::isfinite(B[(size_t)(pl.poison[q].kb * 16 + c) * N + n]);
      for (int i = 0; i < bh; i++) {
        const int32_t row = pl.row_map[((size_t)p * R + s) * bh + i];
        if (row < 0) continue;
        for (int n = 0; n < N; n++) {
          double v = acc[((size_t)s * bh + i) * N + n];
          if (PW)
            for (int t = s + PW; t < R && ((pi.ext_mask >> t) & 1u); t += PW) v += acc[((size_t)t * bh + i) * N + n];
          C[(size_t)row * N + n] = nan[n] ? NAN : v;
        }
      }
    }
  }
  return C;
}

// kind 0: scattered, 1: band with full blocks, 2: hub rows, 3: mixed dense
// and sparse blocks with explicit zeros
void run(int kind, int64_t rows, int64_t cols, int bh, int R, int cls, unsigned seed) {
  std::mt19937_64 rng(seed);
  std::uniform_real_distribution<double> U(0, 1);
  std::vector<int64_t> rp(rows + 1, 0);
  std::vector<int32_t> ci;
  std::vector<float> v;
  for (int64_t r = 0; r < rows; r++) {
    for (int64_t c = 0; c < cols; c++) {
      double d = 0.01;
      if (kind == 1) d = std::llabs(r - c) <= 23 ? 1.0 : 0.0;
      if (kind == 2) d = r % 61 == 5 ? 0.5 : 0.004;
      if (kind == 3) d = (c / 16 + r / 16) % 5 == 0 ? 0.4 : 0.003;
      if (U(rng) < d) {
        ci.push_back((int32_t)c);
        v.push_back(kind == 3 && U(rng) < 0.2 ? 0.0f : (float)(U(rng) * 2 - 1));
      }
    }
    rp[r + 1] = (int64_t)ci.size();
  }
  smat_csr A{rows, cols, (int64_t)ci.size(), rp.data(), ci.data(), v.data(), 0};
  HostBcsr hb;
  Plan g, plain;
  if (build_host_bcsr(A, bh, 16, nullptr, hb) != SMAT_OK || build_plan(hb, R, cls, g, nullptr, true) != SMAT_OK ||
      build_plan(hb, R, cls, plain) != SMAT_OK) {
    check(false, "plan built");
    return;
  }
  const int N = 3;
  std::vector<double> B((size_t)hb.cols_p * N, 0.0);
  for (int64_t k = 0; k < cols; k++)
    for (int n = 0; n < N; n++) B[(size_t)k * N + n] = U(rng) * 2 - 1;
  std::vector<int> seen((size_t)hb.nnzb() * 16, 0);
  const std::vector<double> C = replay(hb, g, R, cls, B, N, &seen);
  for (int64_t k = 0; k < hb.nnzb(); k++)
    for (int c = 0; c < 16; c++) {
      bool nz = false;
      for (int i = 0; i < bh; i++) nz |= hb.val[(size_t)k * bh * 16 + i * 16 + c] != 0.0f;
      check(seen[k * 16 + c] == 1 || (!nz && seen[k * 16 + c] == 0), "every nonzero column once");
    }
  double e = 0, w = 0;
  for (int64_t r = 0; r < rows; r++)
    for (int n = 0; n < N; n++) {
      double s = 0;
      for (int64_t k = rp[r]; k < rp[r + 1]; k++) s += (double)v[k] * B[(size_t)ci[k] * N + n];
      e += (C[r * N + n] - s) * (C[r * N + n] - s);
      w += s * s;
    }
  check(std::sqrt(e / std::max(w, 1e-300)) < 1e-12, "result vs FP64");
  // infinite and NaN values in a few rows of B
  for (int q = 0; q < 6; q++) B[(size_t)(rng() % cols) * N + rng() % N] = q % 2 ? INFINITY : (q % 3 ? -INFINITY : NAN);
  const std::vector<double> X = replay(hb, g, R, cls, B, N, nullptr), Y = replay(hb, plain, R, cls, B, N, nullptr);
  for (int64_t i = 0; i < rows * N; i++)
    check(std::isnan(X[i]) == std::isnan(Y[i]) && (std::isfinite(Y[i]) ? std::fabs(X[i] - Y[i]) < 1e-9 : true) &&
              (std::isinf(Y[i]) ? X[i] == Y[i] : true),
          "same NaN and infinities as the plain plan");
  std::printf("kind %d %ldx%ld bh %d R %d class %d: blocks %ld -> %ld (%zu gathered), tiles %ld -> %ld, MMAs %ld -> %ld\n",
              kind, (long)rows, (long)cols, bh, R, cls, (long)hb.nnzb(), (long)g.stream_blk.size(), g.gcol.size() / 16,
              (long)plain.n_tiles, (long)g.n_tiles, (long)plain.n_groups, (long)g.n_groups);
}

}  // namespace

int main() {
  for (int kind = 0; kind < 4; kind++)
    for (int bh : {16, 32})
      for (int R : {4, 8, 16}) {
        if (bh == 32 && R > 8) continue;
        for (int cls = 0; cls < kPlanClasses; cls++) {
          if (cls == 2 && bh != 16) continue;  // FP8 form: 16-row blocks only
          run(kind, 517, 403, bh, R, cls, 17 * kind + cls);
          if (kind == 2) run(kind, 301, 1511, bh, R, cls, 5);
        }
      }
  run(0, 1, 1, 16, 16, 0, 1);
  run(3, 16, 16, 16, 4, 0, 2);
  std::printf(bad ? "FAIL\n" : "ALL OK\n");
  return bad ? 1 : 0;
}
