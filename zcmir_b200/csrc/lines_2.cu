// The map passes on compile-time lines of 512 to 768 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_2(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 512: *e = run_pass(p, FixedLine<512>{L.tw}, a, st); return true;
        case 576: *e = run_pass(p, FixedLine<576>{L.tw}, a, st); return true;
        case 648: *e = run_pass(p, FixedLine<648>{L.tw}, a, st); return true;
        case 729: *e = run_pass(p, FixedLine<729>{L.tw}, a, st); return true;
        case 768: *e = run_pass(p, FixedLine<768>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
