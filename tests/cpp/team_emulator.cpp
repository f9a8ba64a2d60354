// Host emulation of the generated phases (codegen.h) for one cell: runs the
// text generate_ptx writes on teams of 1 to 128 warps, the last warp
// first, and checks that
//   - no warp reads or writes an item that another warp writes between the
//     same two barriers, and every access lies in the plan's scratch;
//   - the evaluations, factors and solutions are those of plain row-by-row
//     loops bit for bit, for the full and the projection's matrix.
// The dense square's own elimination (a loop of the kernels) is done here by
// plain loops. Reads the mechanism descriptor from a binary file written by
// the test (arrays as int64 count + raw data); argv[2] is the number of
// trailing species with mass 0.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <sstream>
#include <string>
#include <vector>

#include "codegen.h"
#include "layout.h"
#include "symbolic.h"

template <typename T>
std::vector<T> read_array(FILE* f) {
  int64_t n = 0;
  if (fread(&n, sizeof(n), 1, f) != 1) std::exit(3);
  std::vector<T> v(n);
  if (n && fread(v.data(), sizeof(T), n, f) != (size_t)n) std::exit(3);
  return v;
}

enum Op { kLd, kSt, kFma, kMul, kAdd, kSub, kNeg, kMovF, kDiv, kCall, kRet, kBra, kBrx, kBar, kMovS, kSetGe, kAddS };
struct Ins {
  Op op;
  int d = 0, a[3] = {0, 0, 0};
  double imm[3] = {0, 0, 0};
  bool is_imm[3] = {false, false, false}, pred = false;
  int64_t item = 0;
  std::string to;
};
struct Func {
  std::vector<Ins> code;
  std::map<std::string, int> label;
  std::map<std::string, std::vector<std::string>> table;
  int regs = 0;
};

std::map<std::string, Func> parse(const std::string& text) {
  std::map<std::string, Func> fs;
  Func* f = nullptr;
  std::istringstream in(text);
  std::string l;
  while (std::getline(in, l)) {
    const size_t at = l.find(".func ");
    if (at != std::string::npos) {
      const size_t e = l.find('(', at);
      f = &fs[l.substr(at + 6, e - at - 6)];
      continue;
    }
    if (!f) continue;
    while (!l.empty() && (l[0] == '\t' || l[0] == ' ')) l.erase(0, 1);
    if (l.empty() || l[0] == '{' || l[0] == '}' || l.rfind("ld.param", 0) == 0 || l.rfind("st.param", 0) == 0 ||
        l.rfind(".param", 0) == 0 || l.rfind("cvta", 0) == 0 || l.rfind("mov.b64", 0) == 0 ||
        l.rfind("setp.gt", 0) == 0 || l.rfind("setp.ne", 0) == 0 || l.rfind("@%clus", 0) == 0)
      continue;   // a cluster's barrier stands where the block's does
    if (l.rfind(".reg", 0) == 0) {
      if (l.find("%d<") != std::string::npos) f->regs = std::atoi(l.c_str() + l.find("%d<") + 3);
      continue;
    }
    if (l[0] == '$') {
      const size_t c = l.find(':');
      const std::string name = l.substr(0, c);
      const size_t b = l.find(".branchtargets");
      if (b == std::string::npos) {
        f->label[name] = (int)f->code.size();
      } else {
        std::string rest = l.substr(b + 14);
        std::vector<std::string> ts;
        for (char& ch : rest)
          if (ch == ',' || ch == ';') ch = ' ';
        std::istringstream ss(rest);
        for (std::string t; ss >> t;) ts.push_back(t);
        f->table[name] = ts;
      }
      continue;
    }
    Ins i;
    if (l[0] == '@') {
      i.pred = true;
      l = l.substr(l.find(' ') + 1);
    }
    auto operand = [&](int k, const std::string& s) {
      if (s.rfind("%d", 0) == 0) {
        i.a[k] = std::atoi(s.c_str() + 2);
      } else {
        const unsigned long long b = std::strtoull(s.c_str() + 2, nullptr, 16);
        std::memcpy(&i.imm[k], &b, 8);
        i.is_imm[k] = true;
      }
    };
    std::string clean = l;
    for (char& ch : clean)
      if (ch == ',' || ch == ';' || ch == '[' || ch == ']') ch = ' ';
    std::istringstream ss(clean);
    std::vector<std::string> w;
    for (std::string t; ss >> t;) w.push_back(t);
    auto offset = [](const std::string& s) { return (int64_t)std::atoll(s.c_str() + s.find('+') + 1); };
    if (w[0] == "ld.global.f64") { i.op = kLd; i.d = std::atoi(w[1].c_str() + 2); i.item = offset(w[2]); }
    else if (w[0] == "st.global.f64") { i.op = kSt; i.item = offset(w[1]); operand(0, w[2]); }
    else if (w[0] == "call.uni") { i.op = kCall; i.to = w[1]; }
    else if (w[0] == "ret") i.op = kRet;
    else if (w[0] == "bra") { i.op = kBra; i.to = w[1]; }
    else if (w[0] == "brx.idx.uni") { i.op = kBrx; i.to = w[2]; }
    else if (w[0] == "bar.sync") i.op = kBar;
    else if (w[0] == "mov.u32") i.op = kMovS;
    else if (w[0] == "setp.ge.u32") { i.op = kSetGe; i.item = std::atoi(w[3].c_str()); }
    else if (w[0] == "add.u32") i.op = kAddS;
    else {
      i.op = w[0] == "fma.rn.f64" ? kFma : w[0] == "mul.rn.f64" ? kMul : w[0] == "add.rn.f64" ? kAdd
             : w[0] == "sub.rn.f64" ? kSub : w[0] == "neg.f64" ? kNeg : w[0] == "mov.f64" ? kMovF
             : w[0] == "div.rn.f64" ? kDiv : kRet;
      if (i.op == kRet) {
        printf("unknown line: %s\n", l.c_str());
        std::exit(6);
      }
      i.d = std::atoi(w[1].c_str() + 2);
      for (size_t k = 2; k < w.size(); ++k) operand((int)k - 2, w[k]);
    }
    f->code.push_back(i);
  }
  return fs;
}

struct Machine {
  const std::map<std::string, Func>& fs;
  std::vector<double> mem;
  std::vector<int> writer, reader;   // the warp that wrote / read since the barrier (-1 none, -2 several readers)
  int bad = 0;

  Machine(const std::map<std::string, Func>& f, int64_t items) : fs(f), mem(items, NAN) {}

  struct Warp {
    int pc = 0, s = 0;
    bool q = false, done = false;
    std::vector<double> r;
  };

  void touch(int64_t bytes, int w, bool write) {
    const int64_t it = bytes / 256;
    if (bytes % 256 || it < 0 || it >= (int64_t)mem.size()) {
      if (!bad++) printf("access outside the scratch: byte %lld\n", (long long)bytes);
      return;
    }
    if (writer[it] >= 0 && writer[it] != w) {
      if (!bad++) printf("item %lld: warp %d meets warp %d's store\n", (long long)it, w, writer[it]);
    }
    if (write) {
      if (reader[it] != -1 && reader[it] != w && !bad++) printf("item %lld: stored under a reader\n", (long long)it);
      writer[it] = w;
    } else {
      reader[it] = reader[it] == -1 || reader[it] == w ? w : -2;
    }
  }

  // runs one warp to its next barrier or return; pieces run inside
  void advance(const Func& f, Warp& w, int id, int warps) {
    for (;;) {
      const Ins& i = f.code[w.pc++];
      auto v = [&](int k) { return i.is_imm[k] ? i.imm[k] : w.r[i.a[k]]; };
      switch (i.op) {
        case kLd: touch(i.item, id, false); if (bad) return; w.r[i.d] = mem[i.item / 256]; break;
        case kSt: touch(i.item, id, true); if (bad) return; mem[i.item / 256] = v(0); break;
        case kFma: w.r[i.d] = std::fma(v(0), v(1), v(2)); break;
        case kMul: w.r[i.d] = v(0) * v(1); break;
        case kAdd: w.r[i.d] = v(0) + v(1); break;
        case kSub: w.r[i.d] = v(0) - v(1); break;
        case kNeg: w.r[i.d] = -v(0); break;
        case kMovF: w.r[i.d] = v(0); break;
        case kDiv: w.r[i.d] = v(0) / v(1); break;
        case kMovS: w.s = id; break;
        case kSetGe: w.q = w.s >= i.item; break;
        case kAddS: w.s += warps; break;
        case kBra: if (!i.pred || w.q) w.pc = f.label.at(i.to); break;
        case kBrx: w.pc = f.label.at(f.table.at(i.to).at(w.s)); break;
        case kBar: if (warps > 1) return; break;
        case kRet: w.done = true; return;
        case kCall: {
          const Func& g = fs.at(i.to);
          Warp c;
          c.r.assign(g.regs, 0.0);
          c.r[0] = w.r[0];
          advance(g, c, id, warps);
          if (bad) return;
          break;
        }
      }
    }
  }

  void call(const char* name, int warps, double alpha = 1.0) {
    const Func& f = fs.at(name);
    std::vector<Warp> ws(warps);
    for (Warp& w : ws) {
      w.r.assign(f.regs, 0.0);
      w.r[0] = alpha;
    }
    for (;;) {
      writer.assign(mem.size(), -1);
      reader.assign(mem.size(), -1);
      int done = 0;
      for (int w = warps - 1; w >= 0; --w) {
        if (!ws[w].done) advance(f, ws[w], w, warps);
        done += ws[w].done;
        if (bad) std::exit(7);
      }
      if (done == warps) return;
      if (done) {
        printf("%s: a warp returned while others wait\n", name);
        std::exit(8);
      }
    }
  }
};

bool same(double a, double b) { return a == b || (a != a && b != b); }

int main(int argc, char** argv) {
  FILE* fp = fopen(argv[1], "rb");
  if (!fp) return 2;
  auto dims = read_array<int64_t>(fp);                 // n, R, P
  auto react = read_array<int64_t>(fp);
  auto s_indptr = read_array<int32_t>(fp), s_idx = read_array<int32_t>(fp);
  auto s_val = read_array<double>(fp);
  auto rows = read_array<int64_t>(fp), cols = read_array<int64_t>(fp);
  auto j_indptr = read_array<int32_t>(fp), j_idx = read_array<int32_t>(fp);
  auto j_val = read_array<double>(fp);
  fclose(fp);
  const int algebraic = argc > 2 ? std::atoi(argv[2]) : 0;
  std::vector<double> mass(dims[0], 1.0);
  for (int a = 0; a < algebraic; ++a) mass[dims[0] - 1 - a] = 0.0;
  if (algebraic) mass[0] = 2.0;
  fo_mechanism_desc m = {(int32_t)dims[0], (int32_t)dims[1], (int32_t)dims[2], react.data(), s_indptr.data(),
                         s_idx.data(), s_val.data(), (int32_t)rows.size(), rows.data(), cols.data(),
                         j_indptr.data(), j_idx.data(), j_val.data(), mass.data()};
  fo::HostTables t;
  std::string err = fo::build_tables(m, FO_ORDER_AUTO, &t);
  if (!err.empty()) {
    printf("tables: %s\n", err.c_str());
    return 1;
  }
  const fo::GenLayout gl = fo::gen_layout_of(t);
  if (gl.s.items > fo::layout_of(t).items) return 9;
  const int n = t.n, R = t.R, P = t.P;
  fo::GenOptions opt;
  if (argc > 3) opt.tile = std::atoi(argv[3]);
  opt.piece_lines = 300;
  const auto fs = parse(fo::generate_ptx(t, opt));
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> U(0.1, 1.0);
  std::vector<double> k(R), x(n);
  for (double& v : k) v = U(rng);
  for (double& v : x) v = U(rng);
  // plain evaluations
  std::vector<double> F(n), J(t.j_col.size()), d((size_t)R * P, 0.0), r(R);
  auto X = [&](int s) { return x[s]; };
  for (int j = 0; j < R; ++j) {
    double prod = 1.0;
    for (int q = 0; q < P; ++q)
      if (t.react[j * P + q] != n) prod *= X(t.react[j * P + q]);
    r[j] = k[j] * prod;
    for (int a = 0; a < P; ++a) {
      double v = k[j];
      for (int q = 0; q < P; ++q)
        if (q != a && t.react[j * P + q] != n) v *= X(t.react[j * P + q]);
      d[j * P + a] = v;
    }
  }
  for (int i = 0; i < n; ++i) {
    double acc = 0.0;
    for (int q = t.s_ptr[i]; q < t.s_ptr[i + 1]; ++q) acc = std::fma(t.s_val[q], r[t.s_rxn[q]], acc);
    F[i] = acc;
  }
  for (size_t e = 0; e < J.size(); ++e) {
    double acc = 0.0;
    for (int q = t.jt_ptr[e]; q < t.jt_ptr[e + 1]; ++q) {
      const double v = t.jt_val[q] * d[t.jt_idx[q]];
      acc = acc + v;
    }
    J[e] = acc;
  }
  // the adjoint's products, as its table-driven loops scatter them
  const fo::AdjLayout al = fo::adjoint_layout(t, 3);
  std::vector<double> v(n), jbar(J.size()), ybar(n), gref(n, 0.0), wref(R), dbar((size_t)R * P, 0.0), thref(R, 0.0);
  for (double& q : v) q = U(rng) - 0.5;
  for (double& q : jbar) q = U(rng) - 0.5;
  for (double& q : ybar) q = U(rng) - 0.5;
  std::vector<double> yref = ybar;
  for (size_t e = 0; e < J.size(); ++e)
    for (int q = t.jt_ptr[e]; q < t.jt_ptr[e + 1]; ++q)
      dbar[t.jt_idx[q]] = std::fma(-t.jt_val[q], jbar[e], dbar[t.jt_idx[q]]);
  for (int j = 0; j < R; ++j) {
    double w = 0.0;
    for (int e = t.st_ptr[j]; e < t.st_ptr[j + 1]; ++e) w = std::fma(t.st_val[e], v[t.st_sp[e]], w);
    wref[j] = w;
    for (int q = 0; q < P; ++q) {
      const int s = t.react[j * P + q];
      if (s == n) continue;
      gref[s] = std::fma(w, d[j * P + q], gref[s]);
      thref[j] = std::fma(dbar[j * P + q], d[j * P + q], thref[j]);
      for (int q2 = 0; q2 < P; ++q2) {
        if (q2 == q || t.react[j * P + q2] == n) continue;
        double dd = k[j];
        for (int q3 = 0; q3 < P; ++q3)
          if (q3 != q && q3 != q2 && t.react[j * P + q3] != n) dd *= X(t.react[j * P + q3]);
        yref[t.react[j * P + q2]] = std::fma(dbar[j * P + q], dd, yref[t.react[j * P + q2]]);
      }
    }
  }
  for (int warps : {1, 8, 32}) {
    Machine M(fs, al.items);
    for (int j = 0; j < R; ++j) M.mem[gl.s.kc + j] = k[j];
    for (int i = 0; i < n; ++i) {
      M.mem[gl.s.yr + i] = x[i];
      M.mem[al.v + i] = v[i];
      M.mem[al.ybar + i] = ybar[i];
    }
    for (size_t e = 0; e < J.size(); ++e) M.mem[al.jbar + e] = jbar[e];
    M.call("fo_gen_vjp", warps);
    for (int i = 0; i < n; ++i)
      if (!same(M.mem[al.g + i], gref[i])) return printf("vjp %d\n", i), 20;
    for (int j = 0; j < R; ++j)
      if (!same(M.mem[al.w + j], wref[j])) return printf("weight %d\n", j), 21;
    M.call("fo_gen_hvp", warps);
    for (int i = 0; i < n; ++i)
      if (!same(M.mem[al.ybar + i], yref[i])) return printf("hvp %d\n", i), 22;
    for (int j = 0; j < R; ++j)
      if (!same(M.mem[al.w + j], thref[j])) return printf("log k %d\n", j), 23;
  }
  std::vector<double> b(n);
  for (double& v : b) v = U(rng);
  for (int proj = 0; proj < (algebraic ? 2 : 1); ++proj) {
    // plain LU over the full pattern (the projection's with its zeros)
    const double alpha = proj ? 1.0 : 37.5;
    std::vector<double> A((size_t)n * n, 0.0);
    std::vector<char> in((size_t)n * n, 0);
    for (int i = 0; i < n; ++i) {
      for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q) in[(size_t)i * n + t.lu_col[q]] = 1;
      if (!proj || t.mass[i] == 0.0)
        for (int e = t.j_row_ptr[i]; e < t.j_row_ptr[i + 1]; ++e) A[(size_t)i * n + t.j_col[e]] = J[e];
      A[(size_t)i * n + i] += alpha * t.mass[i];
    }
    for (int i = 0; i < n; ++i) {
      for (int kk = 0; kk < i; ++kk) {
        if (!in[(size_t)i * n + kk]) continue;
        const double l = A[(size_t)i * n + kk] * A[(size_t)kk * n + kk];
        A[(size_t)i * n + kk] = l;
        for (int j = kk + 1; j < n; ++j)
          if (in[(size_t)kk * n + j]) A[(size_t)i * n + j] = std::fma(-l, A[(size_t)kk * n + j], A[(size_t)i * n + j]);
      }
      A[(size_t)i * n + i] = 1.0 / A[(size_t)i * n + i];
    }
    std::vector<double> y = b, z = b;
    for (int i = 0; i < n; ++i)
      for (int kk = 0; kk < i; ++kk)
        if (in[(size_t)i * n + kk]) y[i] = std::fma(-A[(size_t)i * n + kk], y[kk], y[i]);
    for (int i = n - 1; i >= 0; --i) {
      for (int j = n - 1; j > i; --j)
        if (in[(size_t)i * n + j]) y[i] = std::fma(-A[(size_t)i * n + j], y[j], y[i]);
      y[i] *= A[(size_t)i * n + i];
    }
    for (int i = 0; i < n; ++i) {
      for (int q = 0; q < i; ++q)
        if (in[(size_t)q * n + i]) z[i] = std::fma(-A[(size_t)q * n + i], z[q], z[i]);
      z[i] *= A[(size_t)i * n + i];
    }
    for (int i = n - 1; i >= 0; --i)
      for (int q = n - 1; q > i; --q)
        if (in[(size_t)q * n + i]) z[i] = std::fma(-A[(size_t)q * n + i], z[q], z[i]);
    for (int warps : {1, 4, 16, 128}) {
      Machine M(fs, gl.s.items);
      for (int j = 0; j < R; ++j) M.mem[gl.s.kc + j] = k[j];
      for (int i = 0; i < n; ++i) M.mem[gl.s.yr + i] = x[i];
      M.call("fo_gen_rhs", warps);
      for (int i = 0; i < n; ++i)
        if (!same(M.mem[gl.s.ft + i], F[i])) return printf("forcing %d\n", i), 10;
      M.call("fo_gen_jac", warps);
      for (size_t e = 0; e < J.size(); ++e)
        if (!same(M.mem[gl.s.negj + e], J[e])) return printf("Jacobian %d\n", (int)e), 11;
      M.call(proj ? "fo_gen_factor_p" : "fo_gen_factor", warps, alpha);
      if (!proj) {
        auto D = [&](int i, int j) -> double& { return M.mem[gl.dense_item(i, j)]; };
        for (int kk = gl.d0; kk < n; ++kk) {
          D(kk, kk) = 1.0 / D(kk, kk);
          for (int i = kk + 1; i < n; ++i) {
            D(i, kk) *= D(kk, kk);
            for (int j = kk + 1; j < n; ++j) D(i, j) = std::fma(-D(i, kk), D(kk, j), D(i, j));
          }
        }
        for (int i = 0; i < n; ++i)
          for (int q = t.lu_row_ptr[i]; q < t.lu_row_ptr[i + 1]; ++q)
            if (!same(M.mem[gl.lu_item[q]], A[(size_t)i * n + t.lu_col[q]]))
              return printf("factor (%d, %d), %d warps\n", i, t.lu_col[q], warps), 12;
      }
      // the square's triangles by plain loops (up: ascending rows)
      auto square = [&](bool up, bool transposed) {
        for (int m = 0; m < n - gl.d0 && !proj; ++m) {
          const int i = up ? gl.d0 + m : n - 1 - m;
          double& xi = M.mem[gl.s.xs + i];
          for (int q = 0; q < m; ++q) {
            const int kk = up ? gl.d0 + q : n - 1 - q;
            xi = std::fma(-M.mem[transposed ? gl.dense_item(kk, i) : gl.dense_item(i, kk)], M.mem[gl.s.xs + kk], xi);
          }
          if (up == transposed) xi *= M.mem[gl.dense_item(i, i)];
        }
      };
      for (int i = 0; i < n; ++i) M.mem[gl.s.xs + i] = b[i];
      M.call(proj ? "fo_gen_solve_p_up" : "fo_gen_solve_up", warps);
      square(true, false);
      square(false, false);
      M.call(proj ? "fo_gen_solve_p_down" : "fo_gen_solve_down", warps);
      for (int i = 0; i < n; ++i)
        if (!same(M.mem[gl.s.xs + i], y[i])) return printf("solve %d, projection %d, %d warps\n", i, proj, warps), 13;
      for (int i = 0; i < n; ++i) M.mem[gl.s.xs + i] = b[i];
      M.call(proj ? "fo_gen_solve_t_p_up" : "fo_gen_solve_t_up", warps);
      square(true, true);
      square(false, true);
      M.call(proj ? "fo_gen_solve_t_p_down" : "fo_gen_solve_t_down", warps);
      for (int i = 0; i < n; ++i)
        if (!same(M.mem[gl.s.xs + i], z[i])) return printf("transposed solve %d, projection %d\n", i, proj), 14;
    }
  }
  printf("n %d square %d of %d blocks\n", n, n - gl.d0, gl.s.nb);
  return 0;
}
