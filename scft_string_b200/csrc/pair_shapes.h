// pair_shapes.h -- which grids have pair-packed kernels (pair.cuh), and the
// launch geometry of those without compile-time sizes.
#pragma once
#include <algorithm>

#include "pair.cuh"

namespace scft {

constexpr int kSmemCta = 227 * 1024 - 128;  // dynamic shared memory a CTA may have, next to the kernels' few static bytes

// slab shapes (m1, m2) and x lengths with kernels
#define PAIR_SLABS(X) X(16, 16) X(24, 24) X(32, 32) X(40, 40) X(48, 48) X(64, 64) X(64, 96) X(80, 80) X(96, 96) X(128, 128)
#define PAIR_AXES(X) X(16) X(24) X(32) X(40) X(48) X(64) X(80) X(96) X(128)

constexpr int kPairTile = 32;  // columns per x tile

// CTAs per slab: one where the slab fits a CTA's shared memory.  Two were slower
// on every shape that fits (one replica step: 64^3 34.2 us with one, 37.1 with
// two; 48^3 22.9 and 27.3; 96^3 84.9 and 91.6).
template <int M1, int M2>
constexpr int kCl = PairSlab<M1, M2, 1>::SMEM <= kSmemCta ? 1 : 2;

inline bool pair_slab_fixed(int m1, int m2)
{
#define X(A, B) \
    if (m1 == A && m2 == B) return true;
    PAIR_SLABS(X)
#undef X
    return false;
}

// CTAs that share a slab
inline int pair_slab_ctas(int m1, int m2)
{
#define X(A, B) \
    if (m1 == A && m2 == B) return kCl<A, B>;
    PAIR_SLABS(X)
#undef X
    return 1;
}

inline bool pair_axis_fixed(int m0)
{
#define X(A) \
    if (m0 == A) return true;
    PAIR_AXES(X)
#undef X
    return false;
}

// n = r1 r2 with both radices available and the larger one as small as it gets
// (at equal size the first the larger: real space and global memory are met with
// more elements per thread); false if there are none
inline bool pair_two_radices(int n, int &r1, int &r2)
{
    static const int rad[] = {
#define X(Q) Q,
        PAIR_RADICES(X)
#undef X
    };
    int best = 1 << 30;
    for (int a : rad)
        for (int b : rad)
            if (a >= b && a * b == n && a < best) {
                best = a;
                r1 = a;
                r2 = b;
            }
    return best < (1 << 30);
}

inline int pair_any_smem(const PairAny &q) { return (q.m1 * q.S + q.m1 + q.m2) * (int)sizeof(cplxd); }
inline int pair_any_pencil_smem(int m0) { return (m0 * kPairTile + m0) * (int)sizeof(cplxd) + (m0 + kPairTile) * (int)sizeof(double); }

inline bool pair_any_plan(int m1, int m2, PairAny &q)
{
    if (m1 < 2 || m2 < 2) return false;
    if (!pair_two_radices(m1, q.ra, q.rb) || !pair_two_radices(m2, q.rc, q.rz)) return false;
    q.m1 = m1;
    q.m2 = m2;
    q.S = m2 | 1;
    q.mag1 = (unsigned)((1ull << 32) / m1) + 1;
    q.mag2 = (unsigned)((1ull << 32) / m2) + 1;
    return pair_any_smem(q) <= kSmemCta;
}

// threads of a slab kernel of such a shape in a launch of `ctas` CTAs: one
// butterfly each in its widest pass, up to 256, or 512 where an SM holds one CTA
// anyway, by its shared memory or because there are no more (one replica step, 256
// and 512 threads: 35x54x45 33.1 and 27.4 us, 60^3 45.2 and 36.5, 112x50x28 38.3
// and 32.7)
inline int pair_any_threads(const PairAny &q, int ctas)
{
    const int n = std::max(std::max(q.m1 * q.rz, q.m1 * q.rc), std::max(q.ra * q.m2, q.rb * q.m2));
    const int most = 2 * (pair_any_smem(q) + 1024) <= 228 * 1024 && ctas > 148 ? 256 : 512;
    return std::min(most, (n + 31) / 32 * 32);
}

inline bool pair_x_radices(int m0, int &r1, int &r2) { return pair_two_radices(m0, r2, r1) && pair_any_pencil_smem(m0) <= kSmemCta; }


// radices of the y transform of a slab, which order its spectra
inline void pair_y_radices(int m1, int m2, int &ra, int &rb)
{
    PairAny q{};
    if (pair_any_plan(m1, m2, q)) {
        ra = q.ra;
        rb = q.rb;
    }
#define X(A, B)                                     \
    if (m1 == A && m2 == B) {                       \
        PairSlab<A, B, kCl<A, B>>::radices(ra, rb); \
    }
    PAIR_SLABS(X)
#undef X
}

// launches of pair_any.cu
int pair_any_setup(int m0, int m1, int m2);
void pair_any_mid(const PropsArgs<double> &a, int nslots, int s, cudaStream_t st);
void pair_any_combine(const PropsArgs<double> &a, int nslots, int s, int mode, int split, cudaStream_t st);
void pair_any_pencil(const PropsArgs<double> &a, int nslots, int s, int both, int nsum, int ra, int rb, cudaStream_t st);

}  // namespace scft
