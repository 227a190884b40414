// fxblock.cuh -- the tables that give a row's columns in the block layout of a sector (fxblock.cu).
#pragma once

#include "fxsum.cuh"

namespace qd {

constexpr int kBlkMaxCross = 8;

struct BlockTables {
  const uint32_t* state;     // the basis in 32 bits
  const int32_t* off;        // 2^highbits: first row of block h
  const uint16_t* rank_low;  // 2^lowbits: rank of l among the low parts of its popcount
  const uint8_t* ldeg;       // 2^lowbits: low targets of l
  const uint16_t* ladj;      // 2^lowbits x lstride: their positions in the block
  const uint8_t* hdeg;       // 2^highbits: high targets of h
  const int32_t* hadj;       // 2^highbits x hstride: first row of each target block
  int lowbits, lstride, hstride, ncross;
  uint32_t cross[3 * kBlkMaxCross];  // support, input pattern, flip
};

BlockTables block_tables(const FxForm& f);

}  // namespace qd
