"""The library's host side on a stand-in CUDA runtime, without a GPU.

tests/fake_cudart.cpp takes the runtime's place: kernels do nothing, but
function attributes belong to a device, launches over a kernel's shared-memory
limit are refused, and every launch, copy, event record and wait is logged with
its stream.  Each case runs in a process of its own.
"""
import ast
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PRELUDE = r"""
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
sys.path.insert(0, sys.argv[2])
import numpy as np
import cumodp_b200 as cm
fake.fake_log.restype = ctypes.c_char_p
L = cm.lib()
P = 469762049

def log():
    return [fake.fake_log(i).decode() for i in range(fake.fake_log_size())]

def root(k):
    return pow(3, (P - 1) >> k, P)  # 3 generates the group

mem = np.zeros(1 << 28, np.int32)  # pages are there once touched
A, B, H = (mem.ctypes.data + (i << 28) for i in range(3))  # 2^26 words each

def product(logn, stream=0):
    n = 1 << (logn - 1)
    cm.fftmul_uni_dev(H, 2 * n - 1, A, n - 1, B, n - 1, P, stream)

def batch(shapes, stream=0):
    d = np.array([n - 1 for n in shapes], np.int32)
    off = np.concatenate([[0], np.cumsum(d.astype(np.int64) + 1)[:-1]])
    cm.fftmul_batch_dev(d, off, A, d, off, B, 2 * off, H, P, stream)

def exact(n, method=0, stream=0):
    rc = L.cumodp_twoconv_mul_i64_dev(n, A, n, B, H, 34, method, stream or None)
    assert rc == 0, rc

def big(n, words, stream=0):
    ow = L.cumodp_twoconv_big_out_words(n, n, 64 * words)
    rc = L.cumodp_twoconv_mul_big_dev(n, A, n, B, words + 1, H, ow, 64 * words, stream or None)
    assert rc == 0, rc
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime_api.h")):
        pytest.skip("no compiler or CUDA headers")
    d = tmp_path_factory.mktemp("fake")
    ver = d / "v.map"
    ver.write_text("libcudart.so.12 { global: *; };\n")
    so = str(d / "libcudart.so.12")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CUDA_INC, "-Wl,-soname,libcudart.so.12",
                        f"-Wl,--version-script={ver}", os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o", so],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]

    def run(code, **env):
        """What the code's last line prints, as a Python value."""
        out = subprocess.run([sys.executable, "-c", PRELUDE + code, so, ROOT], capture_output=True, text=True,
                             timeout=600, env=dict(os.environ, **env))
        assert out.returncode == 0, out.stderr[-2000:]
        return ast.literal_eval(out.stdout.strip().splitlines()[-1])

    return run


@pytest.mark.parametrize("env", [{}, {"CUMODP_ROW_FUSED": "1"}])
def test_every_entry_launches_on_a_second_device(fake, env):
    """Kernels with more than 48 KiB of shared memory run on every device of a process, not only on the first."""
    bad = fake(r"""
bad = []
for dev in (0, 1):
    cm.select_device(dev)
    calls = [("product", product, (k,)) for k in range(5, 26)]
    calls += [("fft", lambda k: cm.fft_uni_dev(A, k, root(k), P, False, 0), (k,)) for k in range(5, 26)]
    calls += [("list", lambda k: cm.list_fft_dev(A, 3, k, root(k), P, True, 0), (k,)) for k in (6, 13, 14, 15, 20)]
    calls += [("fft2d", lambda m, n: cm.fft_bivariate_dev(A, m, root(m), n, root(n), P, False, 0), e)
              for e in ((0, 14), (11, 14), (10, 6), (5, 14))]
    calls += [("bivariate", lambda m, n: cm.bivariate_mul_dev(m, n, A, B, P, 0), e)
              for e in ((5, 6), (12, 12), (10, 14), (11, 13), (11, 14), (12, 10), (2, 5))]
    calls += [("level", lambda l: cm.subproduct_level_dev(l, 3, A, H, P, 0), (l,))
              for l in (1, 16, 300, 513, 1024, 2000, 2048, 5000)]
    calls += [("noalloc", lambda k: cm.fftmul_uni_dev_noalloc(H, (1 << k) - 1, A, (1 << (k - 1)) - 1, B,
                                                             (1 << (k - 1)) - 1, P, 0), (k,)) for k in (8, 13, 14, 17, 20)]
    calls += [("exact", exact, (n,)) for n in (1000, 8192, 40000, 300000)]
    calls += [("big", big, e) for e in ((4, 1), (100, 8), (1024, 16))]
    calls += [("batch", lambda *s: batch(s), e) for e in ((16, 100, 2000), (4096,) * 3, (8192,) * 3, (1 << 17,) * 2)]
    for name, f, args in calls:
        try:
            f(*args)
        except Exception as e:
            bad.append((dev, name, args, str(e)))
print(bad + [l for l in log() if l.startswith("refused")])
""", CUMODP_AUTOTUNE="0", **env)
    assert bad == []


def test_first_batch_of_a_process_times_every_candidate(fake):
    """The autotuner's launches are allowed before the first product of a process has run: a refused one
    counts as a slow one, and the choice is kept (in CUMODP_TUNE_FILE too)."""
    log = fake("""
batch((1 << 19,) * 2)       # 2^20: every split
batch((8192,) * 3)          # 2^14: one CTA per product or three passes
print([l for l in log() if l.startswith(("refused", "launch"))])
""", CUMODP_AUTOTUNE="1")
    assert [x for x in log if x.startswith("refused")] == []
    assert any("k_small_productILi14" in x for x in log)
    assert all(any(f"k_row_mul_fILi{l2}E" in x for x in log) for l2 in range(9, 15))


def test_large_tables_are_made_on_the_device(fake):
    """A prime's or a root's first call uploads no table of more than 2^15 words: the tables of the one-launch
    products and of the four-step rows are 10^5 entries and more, milliseconds on the host."""
    uploads = fake("""
for k in (12, 14, 16):
    product(k)
for k in (15, 20, 24):
    cm.fft_uni_dev(A, k, root(k), P, False, 0)
cm.subproduct_level_dev(2048, 3, A, H, P, 0)
exact(8192)
print([int(l.split()[-1]) for l in log() if l.startswith("copy h2d")])
""")
    assert uploads and max(uploads) <= 1 << 18


STREAMS = r"""
def new_stream():
    s = ctypes.c_void_p()
    fake.cudaStreamCreateWithFlags(ctypes.byref(s), 1)
    return s.value

def fft(k, s):
    cm.fft_uni_dev(A, k, root(k), P, False, s)

calls = {
    "product": lambda s: product(18, s),
    "split_product": lambda s: cm.fftmul_uni_dev(A, 1 << 25, A, (1 << 24), B, 1 << 24, P, s),
    "cyclic": lambda s: L.cumodp_cyclic_mul_dev(4, ctypes.c_void_p(A), ctypes.c_void_p(B), P, ctypes.c_void_p(s)),
    "fft": lambda s: fft(18, s),
    "long_fft": lambda s: fft(26, s),
    "list": lambda s: cm.list_fft_dev(A, 3, 16, root(16), P, False, s),
    "fft2d": lambda s: cm.fft_bivariate_dev(A, 6, root(6), 8, root(8), P, False, s),
    "fft2d_long": lambda s: cm.fft_bivariate_dev(A, 12, root(12), 8, root(8), P, False, s),
    "bivariate": lambda s: cm.bivariate_mul_dev(8, 8, A, B, P, s),
    "bivariate_long": lambda s: cm.bivariate_mul_dev(3, 15, A, B, P, s),
    "exact": lambda s: exact(5000, 0, s),
    "exact_limbs": lambda s: exact(5000, 1, s),
    "exact_long": lambda s: exact(300000, 0, s),
    "big": lambda s: big(64, 8, s),
    "big_long": lambda s: big(1024, 16, s),
    "batch": lambda s: batch((1 << 16,) * 2, s),
    "level": lambda s: cm.subproduct_level_dev(4096, 2, A, H, P, s),
}
"""


NAMES = ["product", "split_product", "cyclic", "fft", "long_fft", "list", "fft2d", "fft2d_long", "bivariate",
         "bivariate_long", "exact", "exact_limbs", "exact_long", "big", "big_long", "batch", "level"]
# these work on the caller's arrays alone
OWN = {"level": "k_monic_level_fixup", "fft2d_long": "k_row_natILi8E"}


def _works(line):
    return line.startswith(("launch", "graph", "copy", "memset"))


def _field(line, what):
    return line.split(what + " ")[1].split()[0]


def _marks(part, s):
    """Events recorded on stream s after the part's last operation there."""
    last = max(i for i, x in enumerate(part) if _works(x) and _field(x, "stream") == s)
    return {_field(x, "event") for x in part[last:] if x.startswith("record") and _field(x, "stream") == s}


def _waits(part, s):
    """Events stream s waits for before any operation of the part."""
    begin = min(i for i, x in enumerate(part) if _works(x))
    return {_field(x, "event") for x in part[:begin] if x.startswith("wait") and _field(x, "stream") == s}


@pytest.mark.parametrize("name", NAMES)
def test_calls_on_two_streams_are_ordered_by_their_scratch(fake, name):
    """A call that uses the library's scratch (or a batch shape's job table) on another stream than the call before
    it gets scratch of its own the first time; from then on its stream waits for an event recorded after that call's
    last operation.  A stream does not wait for itself, and one stream alone is not marked."""
    s1, s2, logs = fake(STREAMS + f"""
f, name = calls[{name!r}], {name!r}
s1, s2 = new_stream(), new_stream()
logs = []
f(s1)  # tables
for s in (s1, s2, s1, s2, s2):
    if name in ("batch", "level"):
        A, B, H = B, H, A  # other operands: the job table is rewritten
    fake.fake_set(b"clear", 0)
    f(s)
    logs.append(log())
print([hex(s1), hex(s2), logs])
""")
    alone, first, third, fourth, fifth = ([x for x in part if OWN.get(name, "(none)") not in x] for part in logs)
    if not any("graph" in x for x in alone):  # (side streams fork and join by events)
        assert not any(x.startswith(("record", "wait")) for x in alone), alone
    begin = min(i for i, x in enumerate(first) if _works(x))
    assert any(x.startswith("malloc") for x in first[:begin]), first
    assert not any(x.startswith("devicesync") for part in logs for x in part)
    assert _marks(first, s2) & _waits(third, s1), (first, third)
    assert _marks(third, s1) & _waits(fourth, s2), (third, fourth)
    assert not _marks(fourth, s2) & _waits(fifth, s2), (fourth, fifth)
    assert not any(x.startswith("malloc") for part in (third, fourth, fifth) for x in part)


@pytest.mark.parametrize("name", ["fft", "bivariate", "exact", "batch"])
def test_a_second_stream_without_memory_waits_for_the_device(fake, name):
    """Where the second stream's copy of the scratch cannot be had, the call waits for the device and shares it."""
    lines = fake(STREAMS + f"""
f = calls[{name!r}]
s1, s2 = new_stream(), new_stream()
f(s1)
A, B, H = B, H, A
L.cumodp_inject_alloc_failures(1)
fake.fake_set(b"clear", 0)
f(s2)
print(log())
""")
    begin = min(i for i, x in enumerate(lines) if _works(x))
    assert any(x.startswith("devicesync") for x in lines[:begin]), lines


def test_host_calls_and_one_stream_share_scratch_by_marks(fake):
    """The library's own stream outlives every call, so what runs on it is marked when another stream asks."""
    lib, s1, logs = fake(STREAMS + """
x = np.ones(1 << 18, np.int32)
s1 = new_stream()
cm.fftmul_uni(x, x, P)
cm.fftmul_uni(x, x, P)
lib = [l.split("stream ")[1].split()[0] for l in log() if l.startswith("launch")][-1]
fake.fake_set(b"clear", 0)
product(19, s1)
print([lib, hex(s1), log()])
""")
    begin = min(i for i, x in enumerate(logs) if _works(x))
    marked = {_field(x, "event") for x in logs[:begin] if x.startswith("record") and _field(x, "stream") == lib}
    assert marked & _waits(logs, s1) and not any(x.startswith("malloc") for x in logs)


@pytest.mark.parametrize("streams", [1, 2])
def test_captured_calls_record_and_wait_for_nothing(fake, streams):
    """Scratch ordering leaves a stream being captured alone: the graph's launches are the caller's to order."""
    lines = fake(STREAMS + f"""
s1, s2 = new_stream(), new_stream()
for s in (s1, s2, s1, s2)[:{3 * streams - 2}]:
    calls["bivariate"](s)
fake.cudaStreamBeginCapture(ctypes.c_void_p(s1), 0)
fake.fake_set(b"clear", 0)
calls["bivariate"](s1)
print(log())
""")
    assert len(lines) == 4 and all(x.startswith("launch") for x in lines)


@pytest.mark.parametrize("what", ["clusters", "pinned_failures"])
def test_host_products_copy_where_the_one_launch_form_is_not_there(fake, what):
    """A host product of 2^16 points reads its operands in place only where the one-launch kernel runs and pinned
    memory is to be had; otherwise its operands are copied to the device, as longer products' are."""
    fast, slow = fake(f"""
x = np.ones(30000, np.int32)
def copies():
    fake.fake_set(b"clear", 0)
    cm.fftmul_uni(x, x, P)
    return [l.split()[1] for l in log() if l.startswith("copy")]
if {what!r} == "clusters":
    fake.fake_set(b"clusters", 0)
    slow = copies(); slow = copies()   # (the first call makes tables)
    cm.select_device(1)
    fake.fake_set(b"clusters", 8)
    fast = copies(); fast = copies()
else:
    fake.fake_set(b"pinned_failures", 2)
    slow = copies(); slow = copies()
    fast = copies()
print([fast, slow])
""")
    assert fast == [] and sorted(slow) == ["d2h", "h2d", "h2d"]


def test_tune_files_of_other_kernels_are_not_used(fake, tmp_path):
    """A choice in CUMODP_TUNE_FILE counts only for the kernels it was timed with."""
    f = tmp_path / "tune"
    f.write_text("0 20 2 14 stand-in/148/sm_10.0\n")  # as written before the key named the kernels
    code = """
batch((1 << 19,) * 2)
print([l for l in log() if l.startswith("launch") and "k_row_mul_f" in l])
"""
    timed = fake(code, CUMODP_AUTOTUNE="1", CUMODP_TUNE_FILE=str(f))
    assert {l2 for l2 in range(9, 15) if any(f"k_row_mul_fILi{l2}E" in x for x in timed)} == set(range(9, 15))
    lines = f.read_text().splitlines()
    assert len(lines) == 2
    again = fake(code, CUMODP_AUTOTUNE="1", CUMODP_TUNE_FILE=str(f))  # and this build's own choice is used
    assert len({x for x in again}) == 1 and f"k_row_mul_fILi{lines[1].split()[3]}E" in again[0]
    assert f.read_text().splitlines() == lines


def test_the_autotuner_times_a_class_at_its_own_size(fake):
    """Whether thousands of short products take a CTA each is timed with a thousand of them: what wins for a few
    hundred loses for them."""
    log = fake("""
batch((4096,) * 4000)   # 2^13
batch((20000,) * 3)     # 2^16
print([l for l in log() if l.startswith("launch")])
""", CUMODP_AUTOTUNE="1")
    grids = {(x.split()[1], tuple(int(v) for v in x.split("grid ")[1].split()[:3])) for x in log}
    assert any("k_small_productILi13" in n and g[0] == 1024 for n, g in grids)
    assert any("k_row_mul_f" in n and g[1] == 4 for n, g in grids)  # three products: a bucket of four


def test_failed_batch_plans_leave_the_byte_count(fake):
    """A batch whose plan runs out of memory half-way gives back what it took, and counts it so."""
    before, after, code = fake("""
L.cumodp_inject_alloc_failures.argtypes = [ctypes.c_int]
batch((4096,) * 3)                      # tables
batch((1 << 16,) * 2)
before = cm.device_bytes_in_use()
fake.fake_set(b"malloc_failure_at", 2)  # the plan's job table is had, its workspace is not
try:
    batch((1 << 16,) * 3)
    code = 0
except cm.CumodpError as e:
    code = e.code
print([before, cm.device_bytes_in_use(), code])
""", CUMODP_AUTOTUNE="0")
    assert code == 0x401 and after == before


def test_refused_cluster_launches_fall_back(fake):
    """Where the set-up found room for a cluster and its launch is refused for resources all the same, the other
    kernels take the product."""
    log = fake("""
product(14)
fake.fake_set(b"refuse_clusters", 1)
fake.fake_set(b"clear", 0)
product(14)
exact(8192)
big(400, 4)
x = np.ones(30000, np.int32)
cm.fftmul_uni(x, x, P)
print(log())
""")
    names = " ".join(x for x in log if x.startswith("launch"))
    assert "k_row_mul_f" in names and "k_residues" in names and "ELi16ELi" not in names  # no 16-CTA form
    assert any(x.startswith("graph") for x in log)
