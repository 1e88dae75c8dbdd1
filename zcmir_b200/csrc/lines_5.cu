// The map passes on compile-time lines of 1944 to 2304 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_5(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 1944: *e = run_pass(p, FixedLine<1944>{L.tw}, a, st); return true;
        case 2048: *e = run_pass(p, FixedLine<2048>{L.tw}, a, st); return true;
        case 2187: *e = run_pass(p, FixedLine<2187>{L.tw}, a, st); return true;
        case 2304: *e = run_pass(p, FixedLine<2304>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
