// Test program for the pivot-list check of bbtc_b200/csrc/layout_check.hpp:
// builds the lists of a graph on the host, plants one named fault and prints
// what the checker says ("OK" when it finds nothing).
//
// usage: pivot_check_harness <graph file> <fault>
// graph file: uint32 n, uint32 P, uint64 m, indptr[n+1], indices[m], cuts[P+1]
#include <cstdio>
#include <string>
#include <vector>

#include "layout_check.hpp"

using namespace bbtc::check;

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* f = std::fopen(argv[1], "rb");
  uint32_t n = 0, P = 0;
  uint64_t m = 0;
  bool ok = f && std::fread(&n, 4, 1, f) == 1 && std::fread(&P, 4, 1, f) == 1 && std::fread(&m, 8, 1, f) == 1;
  std::vector<uint32_t> indptr((size_t)n + 1), indices(m), cuts(P + 1);
  ok = ok && std::fread(indptr.data(), 4, n + 1, f) == n + 1 && std::fread(indices.data(), 4, m, f) == m &&
       std::fread(cuts.data(), 4, P + 1, f) == P + 1;
  if (!ok) return 2;
  std::fclose(f);
  const std::string fault = argv[2];

  Csr g{n, m, indptr.data(), indices.data()};
  std::vector<uint32_t> wptr((size_t)n + 1), pairs, tp, tc;
  row_pairs(g, wptr.data());
  for (uint32_t u = 0; u < n; u++)
    for (uint32_t e = indptr[u]; e < indptr[u + 1]; e++) {
      if (e == indptr[u] || indices[e - 1] / 32 != indices[e] / 32) {
        pairs.push_back(indices[e] / 32);
        pairs.push_back(0);
      }
      pairs.back() |= 1u << (indices[e] % 32);
    }
  Words w{wptr.data(), pairs.data(), pairs.size() / 2};
  transpose(g, tp, tc);
  Csr tr{n, m, tp.data(), tc.data()};

  std::vector<uint32_t> piv, rec(2 * m), crow((m + 31) / 32);
  uint32_t npiv = 0;
  std::vector<uint32_t> last(m, 0);  // per entry: first pivot whose entries end past it
  for (uint32_t v = 0; v < n; v++) {
    uint32_t part = 0;
    while (cuts[part + 1] <= v) part++;
    // the kept part of the row: ids from cuts[part] on
    std::vector<uint32_t> kept;
    for (uint32_t e = indptr[v]; e < indptr[v + 1]; e++)
      if (indices[e] >= cuts[part]) kept.push_back(indices[e]);
    uint32_t end = tp[v];
    for (uint32_t q = tp[v]; q < tp[v + 1]; q++) {
      const uint32_t u = tc[q], word = kept.empty() ? v / 32 : std::min(v / 32, kept[0] / 32);
      if (u < cuts[part + 1]) end = q + 1;
      uint32_t p = wptr[u];
      while (pairs[2 * p] < word) p++;
      rec[2 * q] = p;
      rec[2 * q + 1] = wptr[u + 1];
    }
    const bool is = tp[v + 1] > tp[v] && indptr[v + 1] > indptr[v];
    for (uint32_t q = tp[v]; q < tp[v + 1]; q++) last[q] = is && q >= end ? npiv + 1 : npiv;
    if (!is) continue;
    uint32_t d[8] = {tp[v], end, 0, 0, 0, 0, 0xffffffffu, v};
    if (!kept.empty()) {
      d[2] = wptr[v];
      while (pairs[2 * d[2]] < kept[0] / 32) d[2]++;
      d[3] = wptr[v + 1] - d[2];
      d[4] = kept[0] / 32;
      d[5] = kept.back() / 32 - d[4] + 1;
      d[6] = 0xffffffffu << (kept[0] % 32);
    }
    piv.insert(piv.end(), d, d + 8);
    npiv++;
  }
  for (uint32_t i = 0; i < 8; i++) piv.push_back(i < 2 ? ~0u : 0u);
  for (size_t x = 0; x < crow.size(); x++) crow[x] = last[32 * x];

  const uint32_t k = npiv / 2;  // a pivot in the middle, with entries and a row
  uint32_t* d = &piv[8 * k];
  if (fault == "entries_first") d[0]++;
  else if (fault == "entries_end") d[1]--;
  else if (fault == "vertex") d[7]++;
  else if (fault == "pair") d[2]++;
  else if (fault == "pairs") d[3]--;
  else if (fault == "word") d[4]++;
  else if (fault == "span") d[5]++;
  else if (fault == "bits") d[6] = 0;
  else if (fault == "record_first") rec[2 * d[0]]++;
  else if (fault == "record_end") rec[2 * d[0] + 1]++;
  else if (fault == "index") crow[crow.size() / 2]++;
  else if (fault == "missing") npiv--;
  else if (fault == "surplus") { piv.insert(piv.end(), piv.end() - 8, piv.end()); npiv++; }
  else if (fault == "end_mark") piv[8 * npiv] = (uint32_t)m;
  else if (fault != "none") return 2;

  const std::string why =
      pivots(g, tr, w, Pivots{P, cuts.data(), npiv, piv.data(), rec.data(), crow.data()});
  std::printf("%s\n", why.empty() ? "OK" : why.c_str());
  return 0;
}
