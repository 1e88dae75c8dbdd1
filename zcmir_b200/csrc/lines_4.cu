// The map passes on compile-time lines of 1296 to 1728 points (every 2^a·3^b in between); a
// unit of its own so the instantiations compile in parallel with the others.
#include "passes.cuh"

namespace zc {

bool pass_lines_4(Pass p, const LinePlan& L, const PassArgs& a, cudaStream_t st, cudaError_t* e) {
    switch (L.n) {
        case 1296: *e = run_pass(p, FixedLine<1296>{L.tw}, a, st); return true;
        case 1458: *e = run_pass(p, FixedLine<1458>{L.tw}, a, st); return true;
        case 1536: *e = run_pass(p, FixedLine<1536>{L.tw}, a, st); return true;
        case 1728: *e = run_pass(p, FixedLine<1728>{L.tw}, a, st); return true;
        default: return false;
    }
}

}  // namespace zc
