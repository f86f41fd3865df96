// Tile shapes and epilogue classes of the GEMM kernels, shared by device code and the host's choice between them.
#pragma once

namespace hb {

constexpr int kGemmBM = 128;
constexpr int kGemmBN = 256;
constexpr int kGemmBK = 64;
constexpr int kPairBM = 256;  // rows of a CTA pair's tile (128 per CTA)

enum GemmEpiClass : int { kEpiPlain = 0, kEpiSwiglu = 1, kEpiRope = 2 };

}  // namespace hb
