// gr_single_full.cu -- the single-scene transport kernels for scenes whose arithmetic may
// leave the finite range (class K_FULL: indices outside (1.0005, 8), gain media, inputs that
// are not finite): every term and every channel, clear isotropic stones and the others, the
// environment kind at run time.
#include "gr_single.cuh"

// These scenes ran the extension kernels, which made the short paths of indices near 1 up to
// 1.53 times as long as before the default kernels skipped terms (512 x 512 views of index
// 1.0002 at 2 spp: 283 us then, 417 in the extension kernels, 212 here).
// Resident blocks per SM of the pooled launches, in blocks of 128 threads (2^23 tuples, 9 / 12 /
// 16 blocks: index 9 14.2 / 12.7 / 12.9 ms, a dichroic gain medium 6.80 / 6.88 / 7.36).
constexpr int kFullBlocksClear = 12, kFullBlocks = 9;

namespace grh {

gr_status launch_single_full(int K, const SceneConst &S, const grd::SceneBuffers &B, const grd::LaunchRange &R, float *xyz,
                             cudaStream_t stream, const StagedLaunch *st) {
    constexpr int IC = grd::K_ISO | grd::K_CLEAR;
    if (K & grd::K_CLEAR)
        return st ? launch_staged_mb<IC | grd::K_FULL, kFullBlocksClear>(S, B, R, xyz, stream, st)
                  : launch_plain_k<IC | grd::K_FULL>(S, B, R, xyz, stream);
    return st ? launch_staged_mb<grd::K_FULL, kFullBlocks>(S, B, R, xyz, stream, st)
              : launch_plain_k<grd::K_FULL>(S, B, R, xyz, stream);
}

}  // namespace grh
