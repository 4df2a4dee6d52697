// piece_halves.h -- where a two-pass SGEMM call (gemm_bf16x3.cu) puts its operand
// pieces in its stream's workspace, and whether its split may write them while the
// GEMM of the stream's last such call still reads its own.  Host arithmetic only.
//
// The workspace is [half 0 | half 1], the same for every call of any form (the halves
// move only when the buffer grows, which first drains its stream).  Calls alternate
// between the halves.  Pieces larger than a half take the buffer from its start; the
// call after one of those must not overlap it even where its own half fits, since the
// large pieces reach into both.
#pragma once

#include <stddef.h>

namespace gb {

// Bytes [lo, hi) of the workspace; the half they begin in.
struct PieceRange {
    size_t lo, hi;
    unsigned parity;
};

struct PiecePlace {
    PieceRange at;
    bool apart;   // from the last call's pieces: this call's split may run beside that call's GEMM
};

inline PiecePlace place_pieces(const PieceRange &last, size_t bytes, size_t workspace) {
    const size_t half = workspace / 2 / 256 * 256;
    const bool two_halves = half >= bytes;
    PiecePlace p;
    p.at.parity = two_halves ? last.parity ^ 1u : 0u;
    p.at.lo = p.at.parity * half;
    p.at.hi = p.at.lo + bytes;
    p.apart = two_halves && (p.at.hi <= last.lo || p.at.lo >= last.hi);
    return p;
}

}  // namespace gb
