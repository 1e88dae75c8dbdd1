// The map passes on compile-time lines of 256 to 486 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_1(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 256: *e = run_pass(p, FixedLine<256>{L.tw}, a, st); return true;
        case 288: *e = run_pass(p, FixedLine<288>{L.tw}, a, st); return true;
        case 324: *e = run_pass(p, FixedLine<324>{L.tw}, a, st); return true;
        case 384: *e = run_pass(p, FixedLine<384>{L.tw}, a, st); return true;
        case 432: *e = run_pass(p, FixedLine<432>{L.tw}, a, st); return true;
        case 486: *e = run_pass(p, FixedLine<486>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
