// The strip moment loop of the FP64 form: several Chebyshev steps per launch on a plane
// lattice (gqt_strip.cu).
#pragma once

#include "gqt_forms.h"

namespace gqt {

// Reads `count` offsets j - i of an n-site operator as a lattice of lines (d1 0 when they
// are not): offset k is c1 * d1 + c0 (mod n) with |c1| <= 1, |c0| <= 8, and packed[k] =
// (c0 & 255) | (c1 & 255) << 8.
StripLattice strip_lattice(int n, const int* delta, int count, int* packed);

// The distinct rows of a coded operator: pattern k has len[k] entries, entry m of it of code
// code[k * z + m]; site i has pattern site[i]. At most 256.
struct RowPatterns {
  std::vector<int> len;
  std::vector<uint8_t> code, site;
};

// Whether a loop of h, whose strip lattice is set, may run in strips if its rows are few.
bool strip_possible(gqt_ham* h);

// Fills h's strip_* members but the lattice (at upload); packed and hop: per code its packed
// offset (strip_lattice) and hopping.
gqt_status strip_upload(gqt_ham* h, const RowPatterns& rp, const std::vector<int>& packed,
                        const std::vector<double2>& hop);

// Makes h's records unless they are made (before a capture: it allocates).
gqt_status strip_records(const gqt_ham* h);

// `levels` (at most strip_geo.steps) steps of the FP64 loop on one vector: reads T_{k-2}
// (p2), T_{k-1} (p1) and, unless pair, left; writes the last step's vector to o1 and, if
// levels >= 2, the one before it to o2, which are none of the inputs. Step m's block
// partials go to slab + m * stride, as a deferred step's.
gqt_status strip_steps(const gqt_ham* h, const Op& op, bool pair, int levels, const double2* p2,
                       const double2* p1, double2* o2, double2* o1, const double2* left,
                       double* slab, size_t stride, unsigned* counter);

}  // namespace gqt
