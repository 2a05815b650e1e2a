// Exact factorisation of a multiplier table over 4-bit floats (host side, when a LUT is opened).
//
//     value(i, j) = unit * sum_s F[i][s] * G[j][s],   F, G in {0, +-.5, +-1, +-1.5, +-2, +-3, +-4, +-6}
//
// where value(i, j) = 2^(E >> m) * (2^m + (E & (2^m - 1))) is 2^m times the product 1.i x 1.j the
// table gives (E = carry and mantissa merged, see encode_entry).  The construction walks down the
// rows: value(i, j) = value(0, j) + sum_{s=1..i} D[s][j] with D[s] = row s - row s-1, so F[i][s] is a
// step function of i (c_s below the step, c_s + 1 from it on) and G[j][s] = D[s][j] / unit, which is a
// small integer for any multiplier that is nearly linear in its mantissas.  The steps' lower levels
// c_s are free: sum_s c_s D[s][j] is what is left of row 0 after the remaining slots ("rest"), which
// have a constant F and must be able to hold it.  With c_s = 1 everywhere that sum is row R-1 minus
// row 0, within a few units of row 0 itself for a multiplier that is nearly exact at 2 x 1.j.
// Whatever the search returns is checked against the table entry by entry.
#pragma once
#include <stdint.h>

#include <cmath>
#include <vector>

namespace amsim {

struct CodeTables {
  int slots = 0;               // 0: the table has no such factorisation; else 32, 64 or 128
  int rows_f = 0, rows_g = 0;  // table indices (2^m, or fewer where neighbouring rows are equal)
  int drop_f = 0, drop_g = 0;  // low index bits that do not matter
  double unit = 0;             // of value / 2^m, i.e. of the product of two significands
  std::vector<uint8_t> f, g;   // packed codes, slots / 2 bytes per index, one more row of zeros at the end
};

namespace factor_detail {

constexpr double kLevels[8] = {0, .5, 1, 1.5, 2, 3, 4, 6};
constexpr int kInts[7] = {0, 1, 2, 3, 4, 6, -1};  // integer levels, ended by -1

inline int code_of(double v) {  // 4-bit code of v, -1 if it has none
  for (int c = 0; c < 8; ++c)
    if (std::fabs(v) == kLevels[c]) return v < 0 ? c + 8 : c;
  return -1;
}

struct Spare {
  double a;                // the constant F of the slot
  std::vector<double> b;   // its G per column
};

// The constants a slot may have (bit c: kLevels[c]) for its G to be v divided by the constant.
inline unsigned constants_of(double v) {
  unsigned m = 0;
  for (int c = 1; c < 8; ++c)
    if (code_of(v / kLevels[c]) >= 0) m |= 1u << c;
  return m;
}
// constants_of q quarters; only multiples of a quarter up to 36 have any.
struct ConstantTable {
  unsigned char of[145];
  ConstantTable() {
    for (int q = 0; q <= 144; ++q) of[q] = (unsigned char)constants_of(q / 4.0);
  }
  unsigned operator()(int q) const { return q <= 144 && q >= -144 ? of[q < 0 ? -q : q] : 0; }
};

// Splits rest[j] over at most n constant slots; false if it does not fit.
inline bool split_rest(const std::vector<double>& rest, int n, std::vector<Spare>& out) {
  out.clear();
  bool zero = true;
  for (double r : rest) zero = zero && r == 0;
  if (zero) return true;
  if (n < 1) return false;
  for (int c = 1; c < 8; ++c) {  // one slot: every rest a code times the same constant
    bool ok = true;
    for (double r : rest) ok = ok && code_of(r / kLevels[c]) >= 0;
    if (ok) {
      Spare s{kLevels[c], {}};
      for (double r : rest) s.b.push_back(r / kLevels[c]);
      out.push_back(s);
      return true;
    }
  }
  if (n < 2) return false;
  // several slots: slots of constant 6 take away as much as they can, the last one (constant 1) the remainder
  std::vector<double> left = rest;
  for (int t = 0; t + 1 < n; ++t) {
    Spare s{6, {}};
    for (double& r : left) {
      double best = 0;
      for (int c = 1; c < 8; ++c)
        if (6 * kLevels[c] <= std::fabs(r)) best = kLevels[c];
      if (r < 0) best = -best;
      s.b.push_back(best);
      r -= 6 * best;
    }
    out.push_back(s);
    std::vector<Spare> tail;
    if (split_rest(left, 1, tail)) {
      out.insert(out.end(), tail.begin(), tail.end());
      return true;
    }
  }
  out.clear();
  return false;
}

}  // namespace factor_detail

// entries: encoded bytes (carry << m) + mantissa, row = first operand, 2^m x 2^m, m <= 7.
inline CodeTables factor_table(const uint8_t* entries, int m) {
  using namespace factor_detail;
  CodeTables out;
  const int side = 1 << m;
  auto value = [&](int i, int j) {
    const int e = entries[i * side + j];
    return std::ldexp((double)((1 << m) + (e & (side - 1))), e >> m);
  };
  auto droppable = [&](bool rows, int drop) {  // do the lowest drop + 1 index bits not matter?
    for (int i = 0; i < side; ++i)
      for (int j = 0; j < side; ++j) {
        const int k = (rows ? i : j) >> (drop + 1) << (drop + 1);
        if (entries[i * side + j] != (rows ? entries[k * side + j] : entries[i * side + k])) return false;
      }
    return true;
  };
  int df = 0, dg = 0;
  while (df < m && droppable(true, df)) ++df;
  while (dg < m && droppable(false, dg)) ++dg;
  const int R = side >> df, C = side >> dg;
  std::vector<std::vector<double>> T(R, std::vector<double>(C));
  for (int i = 0; i < R; ++i)
    for (int j = 0; j < C; ++j) T[i][j] = value(i << df, j << dg);

  std::vector<int> step;  // rows that differ from the row above
  for (int i = 1; i < R; ++i)
    if (T[i] != T[i - 1]) step.push_back(i);
  const int nstep = (int)step.size();
  const int slots = nstep + 1 <= 32 ? 32 : nstep + 1 <= 64 ? 64 : nstep + 1 <= 128 ? 128 : 0;
  if (!slots) return out;
  const int spare = slots - nstep;

  for (int ue = 9; ue >= -1; --ue) {  // the largest unit in which every step is a code
    const double unit = std::ldexp(1.0, ue);
    std::vector<std::vector<double>> D(nstep, std::vector<double>(C));
    bool ok = true;
    for (int s = 0; s < nstep && ok; ++s)
      for (int j = 0; j < C && ok; ++j) {
        D[s][j] = (T[step[s]][j] - T[step[s] - 1][j]) / unit;
        ok = code_of(D[s][j]) >= 0;
      }
    if (!ok) continue;
    std::vector<int> level(nstep, 1);  // c_s
    std::vector<Spare> extra;
    auto rest_of = [&]() {
      std::vector<double> r(C);
      for (int j = 0; j < C; ++j) {
        r[j] = T[0][j] / unit;
        for (int s = 0; s < nstep; ++s) r[j] -= level[s] * D[s][j];
      }
      return r;
    };
    bool found = false;
    for (int base = 1; base >= 0 && !found; --base) {
      level.assign(nstep, base);
      found = split_rest(rest_of(), spare, extra);
    }
    if (!found) {
      // two steps on other levels (c, c + 1 both codes: c = -4..3)
      level.assign(nstep, 1);
      const std::vector<double> r0 = rest_of();
      std::vector<double> r(C);
      // Most pairs leave a rest that no slot holds, and a column or two show it: quarters of the unit in integers, stopped
      // there.  (With every column worked out in doubles first, a table of 128 x 128 without a factorisation took one to
      // three seconds to open.)
      const ConstantTable constants;
      std::vector<int> q0(C);
      std::vector<std::vector<int>> step4(nstep, std::vector<int>(C));
      bool quarters = true;
      for (int j = 0; j < C; ++j) {
        quarters = quarters && std::fabs(r0[j]) < 1e6 && r0[j] * 4 == std::floor(r0[j] * 4);
        q0[j] = quarters ? (int)(r0[j] * 4) : 0;
        for (int s = 0; s < nstep; ++s) step4[s][j] = (int)(D[s][j] * 4);  // (codes: whole halves)
      }
      for (int a = 0; a < nstep && !found && quarters; ++a)
        for (int ca = -4; ca <= 3 && !found; ++ca)
          for (int b = a + 1; b < nstep && !found; ++b)
            for (int cb = -4; cb <= 3 && !found; ++cb) {
              unsigned left = 0xFE;
              for (int j = 0; j < C && left; ++j) left &= constants(q0[j] - (ca - 1) * step4[a][j] - (cb - 1) * step4[b][j]);
              if (!left) continue;
              for (int j = 0; j < C; ++j) r[j] = r0[j] - (ca - 1) * D[a][j] - (cb - 1) * D[b][j];
              if (split_rest(r, spare > 1 ? 1 : spare, extra)) {
                level[a] = ca;
                level[b] = cb;
                found = true;
              }
            }
    }
    if (!found) continue;

    std::vector<std::vector<double>> F(R, std::vector<double>(slots, 0.0)), G(C, std::vector<double>(slots, 0.0));
    for (int s = 0; s < nstep; ++s) {
      for (int i = 0; i < R; ++i) F[i][s] = level[s] + (i >= step[s] ? 1 : 0);
      for (int j = 0; j < C; ++j) G[j][s] = D[s][j];
    }
    for (size_t x = 0; x < extra.size(); ++x) {
      for (int i = 0; i < R; ++i) F[i][nstep + x] = extra[x].a;
      for (int j = 0; j < C; ++j) G[j][nstep + x] = extra[x].b[j];
    }
    out.f.assign((size_t)(R + 1) * slots / 2, 0);
    out.g.assign((size_t)(C + 1) * slots / 2, 0);
    bool exact = true;
    auto pack = [&](std::vector<uint8_t>& dst, const std::vector<std::vector<double>>& M) {
      for (size_t i = 0; i < M.size(); ++i)
        for (int s = 0; s < slots; ++s) {
          const int c = code_of(M[i][s]);
          exact = exact && c >= 0;
          dst[i * slots / 2 + s / 2] |= (uint8_t)((c & 15) << (4 * (s & 1)));
        }
    };
    pack(out.f, F);
    pack(out.g, G);
    for (int i = 0; i < R && exact; ++i)
      for (int j = 0; j < C && exact; ++j) {
        double v = 0;
        for (int s = 0; s < slots; ++s) v += F[i][s] * G[j][s];
        exact = v * unit == T[i][j];
      }
    if (!exact) continue;
    out.slots = slots;
    out.rows_f = R;
    out.rows_g = C;
    out.drop_f = df;
    out.drop_g = dg;
    out.unit = unit / side;
    return out;
  }
  return out;
}

}  // namespace amsim
