// cs_host_bands.h — the schedule of a host-buffer run in skewed bands: which
// slabs (rows of a 2D grid, planes of a 3D one) each launch sweeps, and which
// copies of the input it must have waited for. Plain host code.
//
// Group g of the sweeps takes level s (1 .. sweeps) of the slabs from
// g height - align s up to the next group's: it reads nothing that a later
// group computes (align >= radius), and overwrites nothing that one still
// reads, so a group runs all its levels in a row. Every cut is a multiple of
// the kernels' tiles, so that the tiles see the windows of a whole sweep.
//
// The input comes in `chunks` copies, cut where the groups' first levels end
// but for the skew. Each launch and each copy out waits for every chunk that
// holds a point it reads, counted in elements from the layout, so neither a
// last chunk of few slabs (the height is rounded up to the tiles) nor a halo
// whose columns run on in the next row escapes it.
#pragma once
#include "convstencil.h"

#include <algorithm>
#include <vector>

namespace cs {

struct HostBands {
    struct Op {
        enum Kind { kSweep, kSend } kind;
        int chunks;           // copies in that must have arrived: 0 .. chunks - 1
        int level;            // kSweep: level s, from grid (s - 1) % 2 to grid s % 2
        long long from, to;   // kSweep: interior slabs; kSend: elements of the final grid
    };
    std::vector<long long> chunk;  // element boundaries of the copies in
    std::vector<Op> ops;
};

inline HostBands host_bands(const cs_layout &L, int radius, int bands, long long sweeps)
{
    const long long ld = L.pitch[0], slabs = L.extent[0];
    const long long align = L.dims == 2 ? 64 : 8;
    const long long height = ((slabs + bands - 1) / bands + align - 1) / align * align;
    HostBands h;
    h.chunk.push_back(0);
    const long long first = L.origin / ld * ld;  // element where the first interior slab starts
    for (long long s = height; s < slabs; s += height) h.chunk.push_back(first + s * ld);
    h.chunk.push_back(L.elements);
    // Chunks that hold element `last` or one before it.
    auto chunks_to = [&](long long last) {
        int k = 1;
        while (h.chunk[k] <= last) ++k;
        return k;
    };
    // The last element that a sweep of the slabs up to `hi` reads (2D tiles read
    // a window of three rows around them whatever the radius).
    long long reach = L.origin;
    for (int d = 1; d < L.dims; ++d) reach += (L.extent[d] - 1 + radius) * L.pitch[d];
    const long long past = L.dims == 2 ? std::max(radius, 3) : radius;
    auto last_read = [&](long long hi) { return std::min(L.elements - 1, reach + (hi - 1 + past) * ld); };
    const long long groups = (slabs + align * sweeps + height - 1) / height;
    long long sent = 0;
    for (long long g = 0; g < groups; ++g) {
        long long hi = 0;
        for (long long s = 1; s <= sweeps; ++s) {
            const long long lo = std::max(0LL, g * height - align * s);
            hi = std::min(slabs, (g + 1) * height - align * s);
            if (hi > lo) h.ops.push_back({HostBands::Op::kSweep, chunks_to(last_read(hi)), (int)s, lo, hi});
        }
        const long long end = hi == slabs ? L.elements : first + hi * ld;
        if (hi > 0 && end > sent) {
            h.ops.push_back({HostBands::Op::kSend, chunks_to(end - 1), 0, sent, end});
            sent = end;
        }
    }
    return h;
}

}  // namespace cs
