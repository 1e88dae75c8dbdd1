// The map passes on compile-time lines of 2592 to 3888 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_6(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 2592: *e = run_pass(p, FixedLine<2592>{L.tw}, a, st); return true;
        case 2916: *e = run_pass(p, FixedLine<2916>{L.tw}, a, st); return true;
        case 3072: *e = run_pass(p, FixedLine<3072>{L.tw}, a, st); return true;
        case 3456: *e = run_pass(p, FixedLine<3456>{L.tw}, a, st); return true;
        case 3888: *e = run_pass(p, FixedLine<3888>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
