// The map passes on compile-time lines of 48 to 243 points (2^a·3^b in between but 54, 72, 81, 108
// and 162, which run the runtime plan); a unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_0(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 48: *e = run_pass(p, FixedLine<48>{L.tw}, a, st); return true;
        case 64: *e = run_pass(p, FixedLine<64>{L.tw}, a, st); return true;
        case 96: *e = run_pass(p, FixedLine<96>{L.tw}, a, st); return true;
        case 128: *e = run_pass(p, FixedLine<128>{L.tw}, a, st); return true;
        case 144: *e = run_pass(p, FixedLine<144>{L.tw}, a, st); return true;
        case 192: *e = run_pass(p, FixedLine<192>{L.tw}, a, st); return true;
        case 216: *e = run_pass(p, FixedLine<216>{L.tw}, a, st); return true;
        case 243: *e = run_pass(p, FixedLine<243>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
