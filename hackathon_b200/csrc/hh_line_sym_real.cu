// The symmetric line solve for real line coefficients (k^2 real).
#include "hh_line_sym.cuh"

namespace hh {

int launch_sym_real(Plan *p, const double2 *in, double2 *out, int batch, int src_order, const SymMulti *multi) {
    return launch_sym_order<double>(p, in, out, batch, src_order, multi);
}

} // namespace hh
