// schedule.h -- host rules that pick the schedule of a props round; they change the
// order of the work, never a result.
#pragma once

namespace scft {

// Slot groups of a batch of nb replicas where `ngroups` are configured: halved while a
// group of more than two would get fewer than 4 replicas (a launch of 2 or 3 replicas
// leaves most SMs idle: the W+ relaxation runs many such partial batches), and 1 when
// there are fewer than 2 replicas per group.
inline int effective_groups(int ngroups, int nb)
{
    int ng = ngroups;
    while (ng > 2 && nb < 4 * ng) ng /= 2;
    return (ng > 1 && nb >= 2 * ng) ? ng : 1;
}

// The count where none is configured, on a grid of M points: two; on the pair-packed
// kernels the fewest of 2, 4 and 8 whose two groups that run at a time hold no more than
// kLive (spectra, tables and partial result, 64 bytes a point: a third more than the 126
// MB of L2, the largest size that gained) at three replicas a group or more, and two if
// none does.  us per replica step with 2 / 4 / 8 groups, N = 128: 64^3 x12 14.32 / 14.04,
// x14 14.93 / 14.18, x16 15.00 / 14.39 / 14.76, x20 15.19 / 14.70, x24 15.37 / 14.84 /
// 13.90; 48^3 x24 5.92 / 5.69 / 6.63.  Where two groups fit, four lose: 48^3 x16 5.56 /
// 6.08, 64^3 x8 13.57 / 14.83, x10 14.18 / 14.72; where more do not fit either they lose
// or give nothing: 80^3 x12 34.31 / 34.28, x16 34.28 / 34.65, 96^3 x16 59.16 / 59.49 /
// 58.72; 64^3 x11 (three groups would fit, four have fewer replicas) 13.99 / 14.52.
inline int default_groups(bool pair, long long M, int nb)
{
    constexpr double kLive = 169e6;
    if (pair)
        for (int ng = 2; ng <= 8 && (ng == 2 || nb >= 3 * ng); ng *= 2)
            if (nb >= 4 && 2.0 * ((nb + ng - 1) / ng) * 64.0 * (double)M <= kLive) return ng;
    return nb >= 4 ? 2 : 1;
}

// Tile width of an FP32 x pass: 1 wide (2 * tile columns), 0 default; `wide` 1 or 0 says
// so, -1 leaves it to this rule.  Wide where the tiles still fill the SMs four times, for
// their 512-byte rows (16 replicas of 64^3 8.8 us per replica step against 9.2, of 48^3
// 79.7 us a step against 82.0).  Small batches want more blocks (one replica 24.2 us
// wide, 22.1 narrow), and the longer axes spill at twice the butterflies per thread
// (eight replicas of 128^3 109 us wide, 93 narrow).
inline int wide_tiles(int wide, int m0, int ncol, int tile, int spectra, int nslots)
{
    if (wide >= 0) return wide;
    return m0 <= 64 && (ncol + 2 * tile - 1) / (2 * tile) * spectra * nslots >= 4 * 148;
}

}  // namespace scft
