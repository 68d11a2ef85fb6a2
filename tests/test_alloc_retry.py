"""Detection under a memory limit (alloc_retry.hpp compiled as host C++ with a fake
allocator): a list that does not fit beside the kept crossings takes their place, a
string length that does not fit gives back first those, then its own tables; what
fits is allocated once, other errors and a last failure are handed on."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SRC = r"""
#include "alloc_retry.hpp"
#include <cassert>
using namespace lat;
int tries = 0;
long left = 0;
int take(long n)
{
    ++tries;
    if (n > left) return LAT_ERR_NOMEM;
    left -= n;
    return LAT_OK;
}
struct Kept {
    long n;
    bool drop()
    {
        const bool held = n > 0;
        left += n;
        n = 0;
        return held;
    }
};
// the list (`list`) beside the stash; then the length's tables, large or small
int length(long memory, long stash, long list, long large, long small, bool* kept)
{
    left = memory;
    tries = 0;
    Kept st{0};
    if (stash <= left) left -= stash, st.n = stash;
    int rc = alloc_or_release([&] { return take(list); }, [&] { return st.drop(); });
    *kept = st.n > 0;
    if (rc) return rc;
    long tables = large;
    return alloc_or_release([&] { return take(tables); }, [&] { return st.drop(); },
                            [&] {
                                tables = small;
                                return true;
                            });
}
int main()
{
    bool kept;
    assert(length(100, 20, 10, 60, 10, &kept) == LAT_OK && kept && tries == 2);
    assert(length(25, 20, 10, 10, 5, &kept) == LAT_OK && !kept && tries == 3);    // the list in the stash's place
    assert(length(15, 20, 10, 5, 5, &kept) == LAT_OK && !kept && tries == 2);     // no stash from the start
    assert(length(80, 20, 10, 60, 10, &kept) == LAT_OK && kept && tries == 3);    // the tables in the stash's place
    assert(length(50, 20, 10, 60, 10, &kept) == LAT_OK && tries == 4);            // smaller tables
    assert(length(15, 20, 10, 60, 10, &kept) == LAT_ERR_NOMEM && tries == 3);
    assert(length(5, 20, 10, 60, 10, &kept) == LAT_ERR_NOMEM && tries == 1);
    int calls = 0;
    assert(alloc_or_release([&] { ++calls; return LAT_ERR_CUDA; }, [&] { return true; }) == LAT_ERR_CUDA && calls == 1);
    return 0;
}
"""


def test_releases_in_turn(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", f"-I{ROOT / 'axions_gb300' / 'csrc'}", f"-I{ROOT / 'include'}",
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True)
