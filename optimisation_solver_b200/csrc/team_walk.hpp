// team_walk.hpp -- how the threads of an epilogue team go through a CTA's tiles
// (adam_step, gemm.cuh). Compiled for the device there and for the host by its
// test: it holds the order of waits and barriers and nothing of the device.
#pragma once

#ifdef __CUDACC__
#define PDLPGPU_WALK_FN __host__ __device__ __forceinline__
#else
#define PDLPGPU_WALK_FN inline
#endif

namespace pdlpgpu_mlp_impl {

// Tiles first, first + step, ... below `tiles`; tile t has chunks(t) chunks, dealt
// to the teams in turn over the whole walk. Per tile: wait_tile(k), k counting
// the tiles; per chunk of the team wait_chunk(i), i counting them, then
// work(k, c); at the end leave(k). The waits may give up, and then not in
// every thread of the team: agree(ok) tells all of them whether all succeeded,
// and is met by all or none because each tile's result is agreed on before the
// next tile, also by a team without a chunk in it. (Without that, the threads
// whose wait had just succeeded would wait for the others for good.)
template <class Chunks, class WaitTile, class WaitChunk, class Agree, class Work, class Leave>
PDLPGPU_WALK_FN bool team_walk(int first, int step, int tiles, int team, int teams, const Chunks& chunks,
                               const WaitTile& wait_tile, const WaitChunk& wait_chunk, const Agree& agree,
                               const Work& work, const Leave& leave) {
    bool good = true;
    int n = 0, mine = 0;   // chunks of the CTA and of the team
    for (int t = first, k = 0; t < tiles && good; t += step, ++k) {
        const int count = chunks(t);
        good = wait_tile(k);
        bool agreed = false;
        for (int c = 0; c < count; ++c, ++n) {
            if (n % teams != team) continue;
            good = wait_chunk(mine++) && good;
            good = agree(good);
            agreed = true;
            if (!good) break;
            work(k, c);
        }
        if (!agreed) good = agree(good);
        leave(k);
    }
    return good;
}

}  // namespace pdlpgpu_mlp_impl
