// The streaming kernels of layers wider than 6144 x 2048: gate_up with four chunks of 2048 columns (H > 6144), down with one or two.
#include "hmoe_decode_stream.cuh"

namespace hmoe {

void launch_wide_stream(bool grouped, bool down, int grid, const DecodeArgs& a, cudaStream_t st, bool dependent)
{
    if (!down) { if (grouped) launch_stream<true, false, false, 4>(grid, a, st, dependent); else launch_stream<false, false, false, 4>(grid, a, st, dependent); }
    else if (a.I > 2048) { if (grouped) launch_stream<true, false, true, 2, true>(grid, a, st, dependent); else launch_stream<false, false, true, 2, true>(grid, a, st, dependent); }
    else { if (grouped) launch_stream<true, false, true, 1, true>(grid, a, st, dependent); else launch_stream<false, false, true, 1, true>(grid, a, st, dependent); }
}

}  // namespace hmoe
