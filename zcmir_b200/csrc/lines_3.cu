// The map passes on compile-time lines of 864 to 1152 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_3(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 864: *e = run_pass(p, FixedLine<864>{L.tw}, a, st); return true;
        case 972: *e = run_pass(p, FixedLine<972>{L.tw}, a, st); return true;
        case 1024: *e = run_pass(p, FixedLine<1024>{L.tw}, a, st); return true;
        case 1152: *e = run_pass(p, FixedLine<1152>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
