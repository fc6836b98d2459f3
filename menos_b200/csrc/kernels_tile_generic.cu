// Tile-pass instances for any tile width (runtime m, 64-bit amplitude indices),
// with the tile's map and without (TilePass::mapped): 6 brick layers at 24
// qubits in 8-qubit tiles 18.1 ms before the map, 20.0 with it, 17.7 without.
#include "tile_pass.cuh"

namespace mb2 {

int launch_tile_generic(TileLaunch& L) {
    const uint64_t cap = static_cast<uint64_t>(L.sm_count) * 2u;
    L.grid = static_cast<int>(L.ntiles < cap ? L.ntiles : cap);
    return L.mapped ? tile::launch_instance<256, 1, 0, uint64_t, true, true>(L)
                    : tile::launch_instance<256, 1, 0, uint64_t, true, false>(L);
}

}  // namespace mb2
