"""The schedule of host-buffer runs in skewed bands (cs_host_bands.h), replayed on
the CPU over every slab count of a range: no launch reads a point whose copy it
has not waited for, a level that is not there yet or one that has been
overwritten, every slab goes back once and after its last level, and no copy in
is left unwaited for at the end (the caller's array may go then)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "convstencil_gb300", "csrc")

CODE = r"""
#include "cs_host_bands.h"
#include <cstdio>
#include <cstdlib>

static void bad(const char *what, const cs_layout &L, int r, int bands, long long sweeps)
{
    printf("%s: dims %d slabs %lld radius %d bands %d sweeps %lld\n", what, L.dims, L.extent[0], r, bands, sweeps);
    exit(1);
}

static void check(const cs_layout &L, int r, int bands, long long sweeps)
{
    const cs::HostBands h = cs::host_bands(L, r, bands, sweeps);
    const long long slabs = L.extent[0], ld = L.pitch[0];
    if (h.chunk.front() != 0 || h.chunk.back() != L.elements) bad("chunks", L, r, bands, sweeps);
    for (size_t k = 1; k < h.chunk.size(); ++k)
        if (h.chunk[k] <= h.chunk[k - 1]) bad("empty chunk", L, r, bands, sweeps);
    std::vector<long long> level[2] = {std::vector<long long>(slabs, 0), std::vector<long long>(slabs, -1)};
    int waited = 0;
    long long sent = 0, inner = 0;  // inner: first to last point of a slab, halo of r
    for (int d = 1; d < L.dims; ++d) inner += (L.extent[d] - 1 + r) * L.pitch[d];
    for (const auto &op : h.ops) {
        waited = std::max(waited, op.chunks);
        const long long there = h.chunk[waited];  // elements below are on the device
        if (op.kind == cs::HostBands::Op::kSweep) {
            // halo slabs too are read from the grid the copies fill at odd levels
            if ((op.level & 1) && L.origin + (op.to - 1 + r) * ld + inner >= there) bad("early read", L, r, bands, sweeps);
            auto &src = level[(op.level - 1) & 1], &dst = level[op.level & 1];
            for (long long s = std::max(0LL, op.from - r); s < std::min(slabs, op.to + r); ++s)
                if (src[s] != op.level - 1) bad("level", L, r, bands, sweeps);
            for (long long s = op.from; s < op.to; ++s) {
                if (L.origin + s * ld + inner >= there) bad("overwritten by its copy", L, r, bands, sweeps);
                dst[s] = op.level;
            }
        } else {
            if (op.from != sent || op.to <= op.from) bad("send order", L, r, bands, sweeps);
            if (!(sweeps & 1) && op.to > there) bad("early send", L, r, bands, sweeps);
            sent = op.to;
            for (long long s = 0; s < slabs && L.origin + s * ld < op.to; ++s)
                if (level[sweeps & 1][s] != sweeps) bad("send before its last level", L, r, bands, sweeps);
        }
    }
    if (sent != L.elements) bad("not all sent", L, r, bands, sweeps);
    if (waited != (int)h.chunk.size() - 1) bad("copy not waited for", L, r, bands, sweeps);
}

int main()
{
    long long n = 0;
    for (int bands = 2; bands <= 6; ++bands)
        for (long long sweeps : {1, 2, 3, 5, 12, 31}) {
            for (int r : {1, 3})
                for (long long rows = 128 * bands; rows <= 1400; ++rows) {
                    cs_layout L{};
                    L.dims = 2, L.halo = r, L.extent[0] = rows, L.extent[1] = 100, L.pitch[0] = 110, L.pitch[1] = 1;
                    L.origin = 3 * 110 + 4, L.elements = (rows + 6) * 110;
                    check(L, r, bands, sweeps), ++n;
                    L.origin = r * 110 + 1, L.elements = L.origin + (rows - 1 + r) * 110 + 99 + r + 1;  // ends at the last tap
                    if (r == 1) check(L, r, bands, sweeps), ++n;
                    L.origin = 4 * 110, L.elements = (rows + 8) * 110;  // halo columns in the next row
                    check(L, r, bands, sweeps), ++n;
                }
            for (int r : {1, 3})
                for (long long planes = 16 * bands; planes <= 200; ++planes) {
                    cs_layout L{};
                    L.dims = 3, L.halo = r, L.extent[0] = planes, L.extent[1] = 20, L.extent[2] = 30;
                    L.pitch[2] = 1, L.pitch[1] = 38, L.pitch[0] = 38 * 26;
                    L.origin = r * L.pitch[0] + 3 * 38 + 4, L.elements = (planes + 2 * r) * L.pitch[0];
                    check(L, r, bands, sweeps), ++n;
                }
        }
    printf("%lld schedules\n", n);
}
"""


def test_schedule_waits_for_what_it_reads(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "bands.cpp", tmp_path / "bands"
    src.write_text(CODE)
    inc = os.path.join(os.path.dirname(os.path.dirname(CSRC)), "include")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, "-I", inc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
