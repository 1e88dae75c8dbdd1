// The map passes on compile-time lines of 4096 to 8192 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_7(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 4096: *e = run_pass(p, FixedLine<4096>{L.tw}, a, st); return true;
        case 4374: *e = run_pass(p, FixedLine<4374>{L.tw}, a, st); return true;
        case 4608: *e = run_pass(p, FixedLine<4608>{L.tw}, a, st); return true;
        case 5184: *e = run_pass(p, FixedLine<5184>{L.tw}, a, st); return true;
        case 5832: *e = run_pass(p, FixedLine<5832>{L.tw}, a, st); return true;
        case 6144: *e = run_pass(p, FixedLine<6144>{L.tw}, a, st); return true;
        case 6561: *e = run_pass(p, FixedLine<6561>{L.tw}, a, st); return true;
        case 6912: *e = run_pass(p, FixedLine<6912>{L.tw}, a, st); return true;
        case 7776: *e = run_pass(p, FixedLine<7776>{L.tw}, a, st); return true;
        case 8192: *e = run_pass(p, FixedLine<8192>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
