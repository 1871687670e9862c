// The expanded image of an IQ2_XXS tensor: its layout and the two operations that turn it into int8 operands.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace qw4 {

// The kernels that run int8 tensor-core products (the one-kernel decode path and the four-row grouped kernels) read IQ2_XXS from a second
// resident image, made at create (iq2_expand_kernel): every weight as a 2-bit level and a sign bit, laid out for their lanes.  2.06 bits per
// weight become 3.31, and in exchange a lane turns eight weights into MMA operands with shifts, masks and two byte permutes against an
// 8-byte table held in two registers (the codebook and sign look-ups of the packed form cost four shared-memory reads per eight weights
// and bound both kernels).  Decoded values are the same bits.  In the decode kernel a warp spends most of a slice in its MMA loop and HBM
// is a third busy; the bytes still count: with whole 4-bit codes (4.5 bits per weight, one shift and two permutes) four tokens read 65 MB a
// layer instead of 49 and four layers took 162.7 us instead of 153.9.
//
// Block of sixteen rows x 512 columns, 3392 bytes: a slice of a gate/up unit (8 gate rows, 8 up rows) or a down tile.  With row r, half h
// (128 columns) and lane t of the consumer (columns 128 h + 32 j + 8 t .. + 7 of chunk j):
//   [0, 2048)     levels: words at 512 h + 32 r + 8 t; nibble n of word w: column n of chunk 2 w in its low, of chunk 2 w + 1 in its high two bits;
//   [2048, 3072)  signs: word at 256 h + 16 r + 4 t; nibble n, bit j: column n of chunk j;
//   [3072, 3328)  2 * scale + 1 of the chunks: byte at 16 r + 4 h + j;
//   [3328, 3392)  the fp16 super-scales of the two 256-column source blocks: 4 r + 2 (h >> 1).
// The lanes of a warp read consecutive words of each part.
constexpr uint32_t T_IQ2N = 116;                        // not a GGUF type: the expanded image of an IQ2_XXS tensor
constexpr uint32_t IQ2N_LO = 8u | 25u << 8 | 43u << 16 | 60u << 24;                                  // iq2_magnitude(0..3)
constexpr uint32_t IQ2N_HI = (256u - 8u) | (256u - 25u) << 8 | (256u - 43u) << 16 | (256u - 60u) << 24;   // the same, negated
constexpr uint32_t IQ2N_SIGNS = 2048, IQ2N_SCALES = 3072, IQ2N_D = 3328, IQ2N_BLOCK = 3392;
// Permute selectors (level | sign << 2 per nibble) of chunk j.
template <int J>
__device__ __forceinline__ uint32_t iq2n_select(uint2 levels, uint32_t signs) {
    const uint32_t l = J < 2 ? levels.x : levels.y;
    const uint32_t s = J < 2 ? signs << (2 - J) : signs >> (J - 2);
    return ((J & 1 ? l >> 2 : l) & 0x33333333u) | (s & 0x44444444u);
}

}  // namespace qw4
