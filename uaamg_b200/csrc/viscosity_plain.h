// viscosity_plain.h -- which passes of a viscosity level take its plain leaves
// apart (viscosity_march.cuh), by how many it has.  Host, without CUDA.
//
// The passes over both kinds have four CTAs per SM and 128 registers a thread;
// the general kernels, three CTAs with up to 168, hold more of a general leaf's
// loads in flight, which is what a level with few plain leaves needs.  q = A x
// and the first residual gain all the same (leaves without DOFs are skipped).
// Whole solves with viscosity that varies in part of the domain, ms, lists /
// general kernel, by leaves and plain leaves of the level:
//   restriction: 1,107 (245 plain) 6.18 / 6.08; 1,484 (304) 5.32 / 5.26, (0)
//     5.95 / 5.79; 1,948 (584) 6.47 / 6.64, (440) 6.61 / 6.56, (0) 7.30 / 7.16;
//     2,774 (992) 8.77 / 8.79, (420) 9.82 / 9.77, (0) 10.58 / 10.44; 3,836 (674)
//     12.49 / 12.61, (480) 13.09 / 12.97; 5,151 (216) 19.19 / 19.31, (0) 19.68 /
//     19.66; 15,056 over 2,491 (0) 53.4 / 52.6;
//   a colour: 1,107 (218 plain) 4.74 / 4.75, (120) 4.87 / 4.76, (0) 4.98 / 4.80;
//     1,484 (60) 5.77 / 5.83, (0) 5.79 / 5.82; 1,948 (0) 7.16 / 7.18; 2,774 (210)
//     10.20 / 10.24, (70) 10.40 / 10.29, (0) 10.44 / 10.33; 5,151 (0) 19.66 / 19.74.
#pragma once

namespace uaamg {

constexpr int VPLAIN_LARGE = 4096;  // levels of this many leaves: bytes bound both forms
constexpr int VPLAIN_SMALL = 1280;  // levels below: a CTA has one or two leaves in all
constexpr int VPLAIN_RESTRICT = 512;  // plain leaves from which a smaller level's restriction gains

// residual + restriction; plain: leaves plain in every channel
inline bool vplain_restrict(int nl, int plain) {
    return nl >= VPLAIN_LARGE ? plain >= nl / 32 : plain >= VPLAIN_RESTRICT;
}
// a colour of a channel; plain: leaves plain in that channel
inline bool vplain_colour(int nl, int plain) {
    if (nl >= VPLAIN_LARGE) return true;
    return plain >= (nl < VPLAIN_SMALL ? nl / 6 : nl / 32);
}

}  // namespace uaamg
