"""Rules that the kernels launched as programmatic dependents rest on, read
from the sources (a kernel that breaks one may still pass every other test):

- each waits for its predecessor (pdl_wait), also where it returns early;
- one that lets its successor start beside it (pdl_trigger) does so after its
  own wait, so that what ran before its predecessor is complete as well;
- one that holds tensor memory has a barrier between the allocation, which one
  warp makes, and the trigger, which counts for the CTA from its first thread:
  the successor's CTAs take tensor memory too and give it back only after this
  grid has ended."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vring_b200", "csrc")


def _text(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def _sources():
    return {p: _text(p) for p in sorted(glob.glob(CSRC + "/*.cu") + glob.glob(CSRC + "/*.cuh"))}


def _close(src, i):
    """index after the brace that closes the one at i."""
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        j += 1
    return j


def _without_lambdas(body):
    while True:
        m = re.search(r"\[&\]\s*(?:\([^()]*(?:\([^()]*\)[^()]*)*\))?[^{;]*\{", body)
        if not m:
            return body
        body = body[:m.start()] + "LAMBDA" + body[_close(body, m.end() - 1):]


def _bodies(src):
    """name -> body of every __global__ function."""
    out = {}
    for m in re.finditer(r"__global__\s+[^;{]*?\b(k\w+)\s*\((?=[^;]*?\)\s*\{)", src):
        i = src.index("{", m.end())
        out[m.group(1)] = _without_lambdas(src[i:_close(src, i)])
    return out


def _dependents():
    """(name, body) of every kernel that a launch_pdl call may launch."""
    srcs = _sources()
    bodies = {}
    for s in srcs.values():
        bodies.update(_bodies(s))
    names = set()
    for s in srcs.values():
        for m in re.finditer(r"\blaunch_pdl\(([^;]*?);", s):
            arg = re.split(r",\s*(?:dim3|grid|blocks|gr\b|gb\b|std::min)", m.group(1))[0]
            found = [n for n in re.findall(r"\bk\w+", arg) if n in bodies]
            if not found and re.match(r"\s*kern\b", arg):
                before = s[:m.start()]
                at = before.rindex("auto kern =")
                found = [n for n in re.findall(r"\bk\w+", before[at:]) if n in bodies]
            names.update(found)
    return [(n, bodies[n]) for n in sorted(names)]


def test_dependent_kernels_are_found():
    names = [n for n, _ in _dependents()]
    for n in ("k_rhs_march", "k_uppres_march", "k_chunk_tma", "k_chunk_long", "k_lin", "k_dct_w", "k_fft_fwd_s",
              "k_conv3_tc", "k_head", "k_in", "k2d_fcg_pre", "k2d_fcg_xrm", "k_hdnbc"):
        assert n in names, (n, names)


def test_every_dependent_kernel_waits_on_every_way_out():
    for name, body in _dependents():
        assert "pdl_wait();" in body, name
        last = body.rindex("pdl_wait();")
        for m in re.finditer(r"\breturn\s*;", body[:last]):
            assert "pdl_wait();" in body[max(0, m.start() - 120):m.start()], (name, body[m.start() - 120:m.end()])


def test_the_trigger_comes_after_the_wait_and_after_tensor_memory():
    for name, body in _dependents():
        if "pdl_trigger();" not in body:
            continue
        trig = body.index("pdl_trigger();")
        assert "pdl_wait();" in body[:trig], name
        if "tmem_alloc(" in body:
            assert "__syncthreads();" in body[body.index("tmem_alloc("):trig], name
