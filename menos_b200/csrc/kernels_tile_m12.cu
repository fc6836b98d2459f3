// Tile-pass instances for 12-qubit tiles (256 threads, one CTA per SM), lean
// and full variants, with the tile's map and without, as for 11-qubit tiles.
#include "tile_pass.cuh"

namespace mb2 {
namespace {

template <bool MAP>
int launch_map(const TileLaunch& L) {
    if (!L.heavy)
        return L.n_all <= 32 ? tile::launch_instance<256, 1, 12, uint32_t, false, MAP>(L)
                             : tile::launch_instance<256, 1, 12, uint64_t, false, MAP>(L);
    return L.n_all <= 32 ? tile::launch_instance<256, 1, 12, uint32_t, true, MAP>(L)
                         : tile::launch_instance<256, 1, 12, uint64_t, true, MAP>(L);
}

}  // namespace

int launch_tile_m12(TileLaunch& L) {
    const uint64_t cap = static_cast<uint64_t>(L.sm_count);
    L.grid = static_cast<int>(L.ntiles < cap ? L.ntiles : cap);
    return L.mapped ? launch_map<true>(L) : launch_map<false>(L);
}

}  // namespace mb2
