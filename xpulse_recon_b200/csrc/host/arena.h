// arena.h -- offsets of several arrays in one device allocation.  Plain host arithmetic, so that
// the CPU tests check it without a device.
#pragma once

#include <cstdint>

namespace xpr {

constexpr uint64_t kArenaPad = 256;  // what cudaMalloc aligns its allocations to

inline uint64_t arena_round(uint64_t n, uint64_t to) { return (n + to - 1) / to * to; }

// Offsets at[0 .. n) of n parts of bytes[k] bytes whose elements have elem[k] bytes, and their
// total in at[n].  Every part starts on a 256-byte boundary when that fits `available` (true);
// otherwise each one only on a boundary of its own elements (false), which adds nothing to the
// parts' sum when they come in order of falling element size.
inline bool arena_layout(const uint64_t *bytes, const uint64_t *elem, int n, uint64_t available, uint64_t *at)
{
    at[0] = 0;
    for (int k = 0; k < n; ++k) at[k + 1] = arena_round(at[k] + bytes[k], kArenaPad);
    if (at[n] <= available) return true;
    for (int k = 0; k < n; ++k) at[k + 1] = arena_round(at[k] + bytes[k], k + 1 < n ? elem[k + 1] : 1);
    return false;
}

// The same for the two images in flight of the preprocessing: raw pixels twice, a pair of floats,
// preprocessed pixels of `elem` bytes twice.
inline bool staging_layout(uint64_t pixels, uint64_t elem, uint64_t available, uint64_t at[6])
{
    const uint64_t bytes[5] = {pixels * 4, pixels * 4, 8, pixels * elem, pixels * elem}, e[5] = {4, 4, 4, elem, elem};
    return arena_layout(bytes, e, 5, available, at);
}

// A resident reconstruction's arrays: volume, sums, ProjData, preprocessed images (elements of
// `img_elem` bytes) and the separate 16-bit ratio (0 bytes without one).
struct ResidentLayout {
    uint64_t at[6];   // offsets of the five in this order, and their total
    bool at_once;     // all raw images (raw bytes and a pair of floats behind them) fit as well
    uint64_t raw;     // where they start
    uint64_t total;   // with them, when at_once
};

// Raw images that lie together in host memory go up in one copy when they are at most `raw_limit`
// bytes and leave `margin` bytes free: they stay allocated for the whole run, and the device needs
// some room of its own (allocation granularity, kernels loaded at their first launch).  Otherwise
// the images go up one by one, and what that takes for the two in flight stays free here.
inline ResidentLayout resident_layout(const uint64_t bytes[5], uint64_t img_elem, uint64_t pixels, uint64_t raw_bytes,
                                      uint64_t raw_limit, uint64_t margin, uint64_t available)
{
    const uint64_t elem[5] = {4, 4, 4, img_elem, 2};
    ResidentLayout l{};
    uint64_t stage[6];
    staging_layout(pixels, img_elem, ~0ull, stage);
    const bool padded = arena_layout(bytes, elem, 5, available > stage[5] ? available - stage[5] : 0, l.at);
    const uint64_t raw_part = arena_round(raw_bytes, kArenaPad) + 8;
    l.raw = arena_round(l.at[5], kArenaPad);
    l.at_once = padded && raw_bytes && raw_bytes <= raw_limit && l.raw + raw_part + margin <= available;
    l.total = l.at_once ? l.raw + raw_part : l.at[5];
    return l;
}

}  // namespace xpr
