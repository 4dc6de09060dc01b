// CPU build of the integer multiply and divide (phonomena_gb300/csrc/soft_f64.cuh),
// compared with the host's IEEE operations bit for bit.
#include "../phonomena_gb300/csrc/soft_f64.cuh"

using namespace phono;

// kind 0: x / b, 1: x * c, 2: (x * c) / b.  Returns the number of results
// that differ; taken: operands the integer path accepts; exact: how many of
// them needed the exact product or remainder.
extern "C" long soft_check(int kind, const double* x, const double* b, const double* c, long n, long* taken, long* exact) {
  long bad = 0;
  *taken = *exact = 0;
  for (long q = 0; q < n; q++) {
    const SoftRec rb = soft_record(b[q], true, 0), rc = soft_record(c[q], false, 0);
    bool ok;
    const SoftNum s = soft_split(x[q], ok);
    if (!ok || (kind != 1 && !(rb.hi >> 31)) || (kind != 0 && !(rc.hi >> 31))) continue;
    ++*taken;
    const SoftRec& first = kind == 0 ? rb : rc;
    uint64_t p = soft_core(s.hi, s.lo, first.hi, first.lo);
    if (!(p >> 63)) p += p;
    *exact += soft_ambiguous(p);
    auto value = [&] { return b[q]; };
    const double got = kind == 0 ? soft_join(soft_div(s, rb, value))
                                 : kind == 1 ? soft_join(soft_mul(s, rc)) : soft_join(soft_div(soft_mul(s, rc), rb, value));
    const double want = kind == 0 ? x[q] / b[q] : kind == 1 ? x[q] * c[q] : (x[q] * c[q]) / b[q];
    bad += soft_bits(got) != soft_bits(want);
  }
  return bad;
}
