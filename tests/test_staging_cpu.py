"""The staging ring's tables on the host, with a copy that can be made to fail: a table that a later call finds has been copied."""
import ctypes
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc")

FAKE = """
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <utility>
#include <vector>
enum { ZKB_OK = 0, ZKB_EINVAL = -1, ZKB_ECUDA = -2, cudaMemcpyHostToDevice = 1 };
struct zkb_ctx {
    static constexpr int STAGED_TABLES = 32;
    struct StagedTable { size_t pos = 0, n = 0; };
    void* host[64] = {};
    void* device[64] = {};
    void **h_ring = host, **d_ring = device;
    size_t ring_cap = 64, ring_pos = 0;
    StagedTable staged[STAGED_TABLES];
    int staged_next = 0;
    bool on_side = false;
    int stream = 0;
};
static bool copies_fail = false;
static int cudaMemcpyAsync(void* to, const void* from, size_t bytes, int, int) {
    if (copies_fail) return 1;
    memcpy(to, from, bytes);
    return 0;
}
#define ZKB_CUDA(ctx, call) do { if (call) return ZKB_ECUDA; } while (0)
template <class... A> static int set_error(zkb_ctx*, int code, A...) { return code; }
struct DeviceGuard { DeviceGuard(zkb_ctx*) {} };
static int stage_wrap(zkb_ctx* ctx) {
    ctx->ring_pos = 0;
    for (auto& t : ctx->staged) t.n = 0;
    return ZKB_OK;
}
static int stage_reserve(zkb_ctx* ctx, size_t slots) { return ctx->ring_pos + slots > ctx->ring_cap ? stage_wrap(ctx) : ZKB_OK; }
"""
EXPORTS = """
extern "C" zkb_ctx* make() { return new zkb_ctx; }
extern "C" void fail(int on) { copies_fail = on; }
extern "C" int tables(zkb_ctx* c, const uint32_t* const* a, size_t na, const uint32_t* const* b, size_t nb) {
    const std::pair<const uint32_t* const*, size_t> t[2] = {{a, na}, {b, nb}};
    return stage_tables(c, t, 2);
}
// 0: the table is on the device where it is said to be
extern "C" int use(zkb_ctx* c, const void* const* p, int n) {
    void** d = nullptr;
    if (int rc = stage_ptrs(c, p, n, &d)) return rc;
    return memcmp(d, p, n * sizeof(void*)) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    text = open(os.path.join(CSRC, "ctx.cu")).read()
    parts = [re.search(p, text, flags=re.S | re.M).group(0) for p in (r"^static const zkb_ctx::StagedTable\* find_staged.*?(?=^int side_begin)", r"^int stage_tables\(.*?^}\n")]
    d = tmp_path_factory.mktemp("ring")
    src, so = d / "r.cpp", d / "r.so"
    src.write_text(FAKE + "\n".join(parts) + EXPORTS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.make.restype = ctypes.c_void_p
    return lib


def _table(first, n):
    return (ctypes.c_void_p * n)(*range(first, first + n))


@pytest.mark.parametrize("fails", [False, True])
def test_tables_that_are_found_have_been_copied(ring, fails):
    ctx, a, b = ctypes.c_void_p(ring.make()), _table(1000, 5), _table(2000, 9)
    ring.fail(int(fails))
    assert (ring.tables(ctx, a, ctypes.c_size_t(5), b, ctypes.c_size_t(9)) == 0) == (not fails)
    ring.fail(0)
    for _ in range(8):  # ... and past the ring's end
        assert ring.use(ctx, a, 5) == 0 and ring.use(ctx, b, 9) == 0
        assert ring.tables(ctx, _table(3000, 20), ctypes.c_size_t(20), b, ctypes.c_size_t(9)) == 0
