// The module text: its ops, and what is decided from the ops alone before any of them is built.
#pragma once
#include "host_common.h"

#include <algorithm>
#include <cstdlib>
#include <sstream>

namespace tpucb {

using Attrs = std::map<std::string, std::string>;

struct ParsedOp {
  std::string type, name;
  std::vector<std::string> in;
  std::vector<int64_t> shape;
  std::string dtype = "FP32";
  Attrs attrs;
  std::string line; // the text the op was parsed from
  int geti(const char *k, int def = 0) const {
    auto it = attrs.find(k);
    return it == attrs.end() ? def : atoi(it->second.c_str());
  }
  double getf(const char *k, double def = 0) const {
    auto it = attrs.find(k);
    return it == attrs.end() ? def : atof(it->second.c_str());
  }
  std::string gets(const char *k, const char *def = "") const {
    auto it = attrs.find(k);
    return it == attrs.end() ? std::string(def) : it->second;
  }
  // comma-separated integer list attribute (I32ArrayAttr in the reference's op definitions)
  std::vector<int> getl(const char *k) const {
    std::vector<int> v;
    auto it = attrs.find(k);
    if (it == attrs.end()) return v;
    std::stringstream ss(it->second);
    std::string tok;
    while (std::getline(ss, tok, ',')) v.push_back(atoi(tok.c_str()));
    return v;
  }
};

inline std::vector<std::string> split(const std::string &s, char sep) {
  std::vector<std::string> out;
  std::stringstream ss(s);
  std::string tok;
  while (std::getline(ss, tok, sep)) out.push_back(tok);
  return out;
}

inline ParsedOp parse_line(const std::string &line) {
  ParsedOp op;
  op.line = line;
  std::stringstream ss(line);
  std::string tok;
  ss >> op.type;
  while (ss >> tok) {
    auto eq = tok.find('=');
    TPUCB_CHECK(eq != std::string::npos, "module text: token '%s' is not key=value", tok.c_str());
    std::string k = tok.substr(0, eq), v = tok.substr(eq + 1);
    if (k == "name") op.name = v;
    else if (k == "in") op.in = split(v, ',');
    else if (k == "shape") {
      for (auto &d : split(v, ',')) op.shape.push_back(atoll(d.c_str()));
    } else if (k == "dtype") op.dtype = v;
    else op.attrs[k] = v;
  }
  TPUCB_CHECK(!op.name.empty(), "module text: op '%s' has no name", op.type.c_str());
  return op;
}

// Which residual adds run in the epilogue of the convolution that produces their later operand (fuse_residual_add = 2). The launch
// that goes and the operand that is not read again count; the epilogue has room for the add's 14 instructions per four values.
// Behind layers that widen their input: results of 2.5 MiB and more. ResNet-50, us per step alone / with three modules in flight,
// none fused -> by this rule: INT8 batch 8 328.5 / 161.6 -> 314.3 / 155.3, 19 416.6 / 249.1 -> 385.9 / 230.3, 64 729.5 / 621.1 -> 689.7 /
// 561.4, 256 2423 / 2280 -> 2210 / 2011; BF16 (two operands, ReLU) batch 8 498.9 / 233.7 -> 486.9 / 213.6, 32 800.7 / 601.5 -> 779.9 /
// 527.2, 128 2231 / 2174 -> 2088 / 1791. The line is not where the two sides meet: it is that of the epilogue before this one, under
// which smaller results lost 2 to 7 us alone. With this one they gain: every add fused, INT8 batch 1 (none by this rule) 240.4 / 97.8 ->
// 230.7 / 91.7, 3 (none) 273.6 / 114.2 -> 265.0 / 105.7, 8 315.7 / 143.5, 12 340.5 / 187.2 -> 330.7 / 173.1, 19 385.4 / 225.5, 32 484.9 /
// 329.8 against 484.3 / 329.2; BF16 batch 1 (none) 410.9 / 151.9 -> 404.8 / 146.6, 4 446.7 / 174.7 against 450.0 / 177.4. Calls at
// small batches that want them set the option to 1.
// Behind layers that do not widen it (a long K, a short result): up to 4 MiB, where the launch counts (MobileNet-v2, none -> by this
// rule: batch 1 178.2 / 63.8 -> 162.3 / 60.3, 7 213.1 / 104.0 -> 200.3 / 102.1, 32 354.8 / 233.2 -> 335.6 / 234.3, 128 861.0 / 711.6 -> 845.8 /
// 712.5, there every add fused 849.0 / 715.5).
inline bool add_fused_by_size(bool widens, size_t result_bytes) { return widens ? result_bytes >= 5u << 19 : result_bytes <= 4u << 20; }

// The convolutions whose result goes to one residual add only, an add that their epilogue is going to take. They are planned
// without the large tiles of conv_big.cuh, whose epilogue has no add. The conditions are those of fuse_activation_chains, as far
// as the ops tell: a layer kept off the large tiles for an add that then runs by itself would have neither.
// INT8 layers whose time is the loop's keep the large tiles and leave the add to a launch of its own (unless every add is to be
// fused): those of more than 12 K blocks, up to 10 MiB those of 24 and more. Layer and add, us alone / with three modules in
// flight, large tiles and add -> fused:
//   8 blocks (1x1 1024 -> 2048, 7x7) 12 MiB 22.2 / 18.0 -> 18.5 / 18.1, 24 MiB 35.1 / 34.2 -> 34.8 / 33.6; 9 (3x3 64 -> 128, 56x56) 6 MiB 16.6 /
//   10.8 -> 12.0 / 9.8, 12 MiB 22.5 / 17.9 -> 17.4 / 16.5, 24 MiB 37.0 / 33.2 -> 31.2 / 28.9; (128 -> 256, 28x28) 49 MiB 71.5 / 72.7 ->
//   71.0 / 68.9; 12 (1x1 1536 -> 2048) 12 MiB 24.7 / 22.2 -> 22.1 / 22.3;
//   18 blocks, 3x3 at 14x14: 256 -> 512 6 MiB 22.7 / 15.1 -> 19.3 / 14.7, 192 -> 384 9 MiB 30.6 / 25.1 -> 23.3 / 22.5, 256 -> 512 9 MiB
//   24.8 / 21.9 -> 20.9 / 21.8;
//   not: 256 -> 512 12 MiB 31.0 / 27.1 against 28.8 / 28.8, 24 MiB 53.5 / 51.3 against 57.2 / 55.5; 15 blocks (1x1 1900 -> 2048) 24 MiB
//   61.8 / 57.5 against 62.3 / 59.7; 27 (3x3 320 -> 512) 6 MiB 28.5 / 19.2 against 25.2 / 20.6, 12 MiB 39.1 / 34.3 against 40.0 / 40.2.
inline std::set<std::string> residual_add_tails(const std::vector<ParsedOp> &ops, const std::map<std::string, const ParsedOp *> &by_name,
                                                const std::map<std::string, int> &n_uses, int fuse, int max_batch) {
  std::set<std::string> tails;
  for (const ParsedOp &add : ops) {
    const bool bf16 = add.dtype == "BF16";
    if (fuse == 0 || add.type != "eltwise_add" || !(bf16 || add.dtype == "INT8")) continue;
    std::vector<const ParsedOp *> from; // the operands that are results
    for (auto &nm : add.in) {
      auto it = by_name.find(nm);
      if (it != by_name.end() && it->second < &add) from.push_back(it->second);
    }
    if (from.size() != 2 || from[0] == from[1]) continue;
    const ParsedOp &conv = *std::max(from[0], from[1]), &other = *std::min(from[0], from[1]);
    if (conv.type != "conv_2d" && conv.type != "deconv_2d") continue;
    if (other.type == "reshape" || conv.geti("g", 1) != 1 || conv.geti("do_relu", 0) || n_uses.at(conv.name) != 1) continue;
    if (conv.dtype != add.dtype || other.dtype != add.dtype || conv.shape != add.shape || other.shape != add.shape) continue;
    bool ones = true;
    std::stringstream coeffs(add.gets("coeff"));
    for (std::string c; std::getline(coeffs, c, ',');) ones = ones && atof(c.c_str()) == 1.0;
    if (bf16 && !(add.geti("do_relu", 0) && ones)) continue;
    if (fuse == 2) {
      auto src = conv.in.empty() ? by_name.end() : by_name.find(conv.in[0]);
      if (src == by_name.end()) continue;
      auto extent = [](const ParsedOp &op, size_t k) { return k < op.shape.size() ? op.shape[k] : (int64_t)1; };
      const int pitch = round_up((int)extent(conv, 1), 16), in_pitch = round_up((int)extent(*src->second, 1), 16);
      const size_t bytes = (size_t)extent(conv, 0) * max_batch * extent(conv, 2) * extent(conv, 3) * pitch * (bf16 ? 2 : 1);
      if (!add_fused_by_size(pitch > in_pitch, bytes)) continue;
      const int k_blocks = conv.geti("kh", 1) * conv.geti("kw", 1) * ((in_pitch + 127) / 128);
      if (!bf16 && k_blocks > 12 && (k_blocks >= 24 || bytes > 10u << 20)) continue;
    }
    tails.insert(conv.name);
  }
  return tails;
}

} // namespace tpucb
