// How the CTAs of dq_stream.cu share its units of work, for the kernel, the host code that sizes the workspace, and the tests.
#ifndef NNF_STREAM_SHARES_H
#define NNF_STREAM_SHARES_H

#ifdef __CUDACC__
#define NNF_HD __host__ __device__ __forceinline__
#else
#define NNF_HD inline
#endif

namespace nnf
{
// tiles x KU units, tile by tile, in contiguous shares: the first `rem` CTAs have lo + 1 of them, the others lo (at least one).
struct StreamShares
{
    int tiles, KU, ctas, lo, rem;

    NNF_HD void set(int tiles_, int KU_, int most_ctas)
    {
        tiles = tiles_, KU = KU_;
        ctas = tiles * KU < most_ctas ? tiles * KU : most_ctas;
        lo = tiles * KU / ctas, rem = tiles * KU % ctas;
    }
    NNF_HD int begin(int cta) const { return cta * lo + (cta < rem ? cta : rem); }
    NNF_HD int units(int cta) const { return lo + (cta < rem ? 1 : 0); }
    // the CTA whose share holds unit u
    NNF_HD int owner(int u) const
    {
        const int more = rem * (lo + 1); // units of the shares with one more
        return u < more ? u / (lo + 1) : rem + (u - more) / lo;
    }
    NNF_HD bool any_shared() const { return tiles % ctas != 0; } // is a tile shared?
    // Where a CTA leaves its sums of a tile that it shares.  From one part of a tile to the next the CTA, the tile or both go up by
    // one, so that their sum tells parts apart; with more tiles than CTAs a CTA shares its first tile and its last at most.
    NNF_HD int slot(int cta, int tile) const { return tiles <= ctas ? cta + tile : 2 * cta + (begin(cta) >= tile * KU ? 0 : 1); }
    NNF_HD int slots() const { return !any_shared() ? 0 : tiles <= ctas ? ctas + tiles - 1 : 2 * ctas; }
};
} // namespace nnf

#endif
