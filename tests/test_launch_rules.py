"""Rules by which launches are cut, checked on the host: compiled from the kernels' own headers."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "attention.cuh"
#include "row_parts.cuh"
using namespace carat_b200;
extern "C" int part_columns(int width, int parts) { return row_part_columns(width, parts); }
extern "C" int parts_of(int rows, int width, int resident, int sms) {
  return geglu_parts(rows, width, resident != 0, sms);
}
extern "C" int chunk(int requests, int kv_heads, int rows, int sms) {
  return chunk_rows(requests, kv_heads, rows, sms);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None or shutil.which("nvcc") is None:
        pytest.skip("no g++ or no CUDA headers")
    cuda_home = os.environ.get("CUDA_HOME", os.path.dirname(os.path.dirname(shutil.which("nvcc"))))
    folder = tmp_path_factory.mktemp("rules")
    source, library = folder / "rules.cpp", folder / "rules.so"
    source.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "carat_b200", "csrc"), "-I",
                    os.path.join(cuda_home, "include"), str(source), "-o", str(library)],
                   check=True, timeout=120)
    return ctypes.CDLL(str(library))


@pytest.mark.parametrize("sms", [148, 132])
@pytest.mark.parametrize("resident", [0, 1])
def test_geglu_parts_cover_the_row_and_stay_few(rules, resident, sms):
    # 8 x 1031 and 8 x 2687 have no divisor near the wanted part count.
    for width in (8, 512, 8184, 8192, 8 * 1031, 16 * 1031, 21504, 8 * 2687, 43008, 65536 + 8):
        for rows in (1, sms, sms + 1, 2048):
            parts = rules.parts_of(rows, width, resident, sms)
            assert 1 <= parts <= max(2, -(-width // 8192)), (width, rows)
            span = rules.part_columns(width, parts)
            assert span % 8 == 0 and (parts - 1) * span < width <= parts * span, (width, rows)
            if resident:
                assert rows * parts <= 2 * sms or parts == 1
            elif rows > sms:
                assert span <= 8192


@pytest.mark.parametrize("sms", [148, 132])
def test_a_cut_context_leaves_every_chunk_an_sm(rules, sms):
    for kv_heads in (1, 4, 16):
        for requests in (1, 2, 5, 9, 18, 20, 24, 37, 1024):
            for rows in (1, 255, 257, 513, 905, 1024, 1025, 3000, 5005, 8192, 30000, 262144):
                chunk = rules.chunk(requests, kv_heads, rows, sms)
                assert chunk % 128 == 0 and (256 <= chunk <= 512 or chunk == 1024)
                if chunk != 1024:
                    chunks = -(-rows // chunk)
                    assert rows > 512
                    if chunks == 2 and chunk > 256:
                        assert rows > 640 and requests * kv_heads * 2 <= sms * 5 / 6
                    assert requests * kv_heads * chunks <= sms, (requests, kv_heads, rows)
    assert rules.chunk(20, 4, 905, sms) == 1024      # two chunks a request: 160 on 148 SMs
    assert rules.chunk(18, 4, 905, sms) == 1024      # two chunks a request, on too many SMs
    assert rules.chunk(13, 4, 905, sms) == 512 and rules.chunk(13, 4, 625, sms) == 1024
    assert rules.chunk(8, 4, 325, sms) == 1024
    assert rules.chunk(1, 4, 905, sms) == rules.chunk(5, 4, 565, sms) == 256
