"""Host planning (hs_runtime.cu): what one launch sequence may index, and what its
workspace holds.  A program linked with the library plans and carves without a GPU."""

import subprocess

import pytest

import _cpp
from conftest import ROOT
from test_pull_pieces import cuda_include

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <string>
#include "hs_internal.h"
using namespace hs;
int main(int argc, char **argv)
{
    const std::string what = argv[1];
    Context ctx;
    ctx.sm_count = 152;
    auto arg = [&](int i) { return (size_t)std::stoull(argv[i]); };
    if (what == "batch") {  // curve, window rule (0: none), then pairs (count, points)
        const int curve = (int)arg(2);
        if (arg(3))
            ctx.rules[curve].push_back(WindowRule{0, size_t(1) << 40, (int)arg(3)});
        std::vector<size_t> sizes;
        for (int i = 4; i + 1 < argc; i += 2)
            sizes.insert(sizes.end(), arg(i), arg(i + 1));
        const BatchPlan p = make_batch_plan(ctx, curve, sizes.data(), (uint32_t)sizes.size());
        std::printf("%d %llu %llu %u %zu %u\n", (int)p.fits(), (unsigned long long)p.entries_bound,
                    (unsigned long long)p.buckets, p.ba_rounds, batch_bytes(p), p.msms[0].c);
    } else if (what == "indexed") {  // window, count, points
        const std::vector<size_t> sizes(arg(3), arg(4));
        const BatchPlan p = make_indexed_plan(ctx, 0, sizes.data(), (uint32_t)sizes.size(), (int)arg(2));
        std::printf("%d\n", (int)p.fits());
    } else if (what == "fixed") {  // generators, window, count
        const size_t chunk = fixed_chunk(arg(2), (int)arg(3), arg(4));
        const BatchPlan p = make_fixed_plan(0, arg(2), (int)arg(3), (uint32_t)chunk);
        std::printf("%zu %d\n", chunk, (int)p.fits());
    } else if (what == "chunks") {  // generators, window, count, rounds
        ctx.ba_set[0] = true;
        ctx.ba_rounds[0] = (uint32_t)arg(5);
        const size_t n = arg(2), count = arg(4), chunk = fixed_chunk(n, (int)arg(3), count);
        for (size_t j = 0; j < count; j += chunk) {
            DeviceArena a;  // nothing is read or written: the buffers are only laid out
            a.base = reinterpret_cast<char *>(256);
            a.cap = fixed_workspace(ctx, 0, n, (int)arg(3), count) + 1024;
            BatchBuffers b;
            std::printf("%d", (int)carve(a, fixed_plan(ctx, 0, n, (int)arg(3), (uint32_t)std::min(chunk, count - j)), b));
            a.base = nullptr;
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    inc = cuda_include()
    if inc is None or not (_cpp.LIBDIR / "libhelioselene_gb300.so").exists():
        pytest.skip("CUDA runtime headers or the library not found")
    d = tmp_path_factory.mktemp("plans")
    (d / "plans.cpp").write_text(PROGRAM)
    subprocess.run([_cpp.gxx(), "-std=c++17", "-O1", f"-I{inc}", f"-I{ROOT / 'helioselene_gb300' / 'csrc'}",
                    str(d / "plans.cpp"), "-o", str(d / "plans"), f"-L{_cpp.LIBDIR}", "-lhelioselene_gb300",
                    f"-Wl,-rpath,{_cpp.LIBDIR}"], check=True, capture_output=True, text=True)

    def run(*args):
        return subprocess.run([str(d / "plans"), *map(str, args)], check=True, capture_output=True, text=True).stdout

    return run


# the last two: counts whose product with the buckets of an MSM wraps at 2^32
@pytest.mark.parametrize("window,count,n,fits", [
    (0, 1, 1, 1), (0, 1024, 65536, 1), (0, 1000000, 1, 1), (0, 1 << 11, 1 << 20, 0), (20, 315, 1, 1), (20, 316, 1, 0),
    (20, 640, 1, 0), (0, 5200000, 1, 0)])
def test_batches_that_one_launch_sequence_indexes(plan, window, count, n, fits):
    got, entries, buckets = plan("batch", 0, window, count, n).split()[:3]
    assert int(got) == fits
    assert fits == (int(entries) < 2**31 and int(buckets) < 2**31)


@pytest.mark.parametrize("window,count,n,fits", [(12, 1024, 4096, 1), (16, 65535, 1, 1), (16, 65536, 1, 0),
                                                (16, 131073, 1, 0), (16, 7000, 8192, 1), (16, 7800, 8192, 0)])
def test_indexed_batches(plan, window, count, n, fits):
    assert int(plan("indexed", window, count, n)) == fits


@pytest.mark.parametrize("n,window,count,chunk", [(1, 6, 100, 100), (228, 9, 8192, 8192), (1 << 20, 20, 4096, 39),
                                                 (1, 20, 8192, 4095), (1, 16, 70000, 65535), (100, 16, 140000, 65535)])
def test_fixed_base_chunks(plan, n, window, count, chunk):
    got, fits = plan("fixed", n, window, count).split()
    assert (int(got), int(fits)) == (chunk, 1)



# curve 1 takes two rounds by default; sparse lists (at most 4 entries a bucket) none, and
# without them an MSM of three points takes less than the 128 KB that 33 windows of 128
# buckets take
@pytest.mark.parametrize("count,n,rounds", [(8192, 200, 2), (4096, 64, 0), (281073, 3, 0), (800000, 3, 0)])
def test_rounds_and_workspace_of_many_small_msms(plan, count, n, rounds):
    fits, _, _, got, bytes_, _ = plan("batch", 1, 0, count, n).split()
    assert (int(fits), int(got)) == (1, rounds)
    assert n > 3 or int(bytes_) < count * 128000, bytes_


# chunks of 1024 commitments whose last one has groups half the size
@pytest.mark.parametrize("rounds", [0, 1, 2])
@pytest.mark.parametrize("n,window,count", [(26214, 13, 1024 + 1023), (26214, 13, 2048), (5000, 10, 4129 + 4095),
                                            (228, 9, 200000)])
def test_every_chunk_of_commitments_has_its_workspace(plan, n, window, count, rounds):
    out = plan("chunks", n, window, count, rounds)
    assert len(out) >= 2 and set(out) == {"1"}, out


# many MSMs of 600 points: 7 bits by default, more where that exceeds what is indexed
@pytest.mark.parametrize("count,c,fits", [(96000, 7, 1), (97000, 8, 1), (130000, None, 0)])
def test_widths_at_the_limit_of_the_entries(plan, count, c, fits):
    got, entries, _, _, _, width = plan("batch", 0, 0, count, 600).split()
    assert int(got) == fits and (c is None or (int(width) == 7 if c == 7 else int(width) >= c))
    assert not fits or int(entries) < 2**31
