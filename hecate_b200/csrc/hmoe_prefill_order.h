// When the converting warps of the grouped GEMMs (hmoe_prefill.cu) have to wait for one another before they wait for codes; apart from them so that a
// host program can walk through it.
//
// Two groups of warps take a tile's stages in turn (stage t is group t & 1's) and read the packed codes from PF_NCODE slots that one warp fills
// in the order of the stages: a stage takes one slot, with the int8 shared expert two. A wait for codes names a use of its slot by the use's
// parity, which tells it from the use before only once that one is known to be in. It is if this group has itself waited for it: as long as every
// stage takes one slot (PF_NCODE is even). Behind an item whose stages took two, the use before may have been the other group's, so the warps first wait until
// all of them have come that far; from the next item's fifth slot on the uses before are the group's own again. An int8 stage waits
// for its operand slot before its codes: the stages up to t - 2 are multiplied then, so their codes are in, and t - 1 took two slots at most.
#pragma once
#include <cstdint>

namespace hmoe {

constexpr uint32_t PF_NCODE = 4;

struct CodeOrder
{
    bool after_i8 = false;                      // the item before was one of the int8 format
    uint32_t crossings = 0;                     // how often the warps have waited for one another
#ifdef __CUDACC__
    __host__ __device__ __forceinline__
#endif
    bool wait_first(bool i8)                    // called once per item
    {
        const bool first = after_i8 && !i8;
        after_i8 = i8;
        crossings += first;
        return first;
    }
};

}  // namespace hmoe
