"""Which library calls the drainage program makes of its options: the program
compiled against a stand-in for the library that prints them."""
import os
import subprocess

import pytest

STANDIN = r"""
#include <cstdio>
#include "cageo.h"
extern "C" {
const char* cageo_last_error_string(void) { return "refused"; }
int cageo_filter_radius(float, float) { return 3; }
cageo_status cageo_read_header(const char*, cageo_raster_info* i) {
  i->ncols = 8; i->nrows = 6; i->cellsize = 10.0f; i->nodata_value = -9999.0f;
  return CAGEO_OK;
}
cageo_status cageo_read_raster(const char*, float*, size_t) { return CAGEO_OK; }
cageo_status cageo_write_raster(const char*, const float*, size_t) { return CAGEO_OK; }
cageo_status cageo_write_jpeg(const char*, const uint8_t*, int, int, int) { return CAGEO_OK; }
cageo_status cageo_pipeline_create(cageo_pipeline**, const cageo_pipeline_config*, const float*,
                                   const float*) { return CAGEO_OK; }
cageo_status cageo_pipeline_set_batch(cageo_pipeline*, int k) {
  std::printf("set_batch %d\n", k);
  return k >= 1 && k <= 64 ? CAGEO_OK : CAGEO_ERR_ARGUMENT;
}
cageo_status cageo_pipeline_run(cageo_pipeline*, uint32_t first, int count) {
  std::printf("run %u %d\n", first, count);
  return CAGEO_OK;
}
cageo_status cageo_pipeline_load(cageo_pipeline*, const char*, uint32_t*) { return CAGEO_OK; }
cageo_status cageo_pipeline_save(cageo_pipeline*, const char*, uint32_t) { return CAGEO_OK; }
cageo_status cageo_pipeline_counts(cageo_pipeline*, float*) { return CAGEO_OK; }
cageo_status cageo_pipeline_counts_bytes(cageo_pipeline*, uint8_t*) { return CAGEO_OK; }
cageo_status cageo_pipeline_stats(cageo_pipeline*, int64_t*, int) { return CAGEO_OK; }
void cageo_pipeline_destroy(cageo_pipeline*) {}
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from cageo_gb300 import _build
    d = tmp_path_factory.mktemp("cli")
    (d / "standin.cpp").write_text(STANDIN)
    out = str(d / "drainage")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", _build.INCLUDE, "-I",
                    os.path.join(_build.CUDA_HOME, "include"), "-o", out,
                    os.path.join(_build.CSRC, "drainage_main.cpp"), str(d / "standin.cpp")],
                   check=True)
    return out


@pytest.mark.parametrize("args, calls", [
    ([], ["run 0 7"]),                                        # the grid's size decides
    (["--batch", "1"], ["set_batch 1", "run 0 7"]),           # one at a time, no stacks
    (["--batch=4"], ["set_batch 4", "run 0 7"]),
    (["--batch", "1", "--fill", "exact"], ["set_batch 1", "run 0 7"]),
])
def test_batch_option(program, tmp_path, args, calls):
    r = subprocess.run([program, "-i", "7", "--seed", "1", "-o", "x.bin", *args], cwd=tmp_path,
                       capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    made = [s for s in r.stdout.splitlines() if s.startswith(("set_batch", "run"))]
    assert made == calls


@pytest.mark.parametrize("value", ["0", "65", "x"])
def test_batch_refused(program, tmp_path, value):
    r = subprocess.run([program, "-i", "7", "--batch", value], cwd=tmp_path, capture_output=True,
                       text=True, timeout=60)
    assert r.returncode == 1 and "batch: refused" in r.stderr
