"""Kernels that start before the one ahead of them has ended (those that call
pdl_wait) read what it writes only after the wait.

A load through a kernel argument declared __restrict__ does not have that
order: the declaration promises that nothing else writes the data while the
kernel runs, so the compiler may move the load above the wait, whose memory
clobber covers only data that others can reach.  Such a kernel may therefore
declare __restrict__ only on what is written before every kernel that can still
run beside it: the tables listed in SETTLED, per kernel where the reason is
its own.  The order cannot be observed by running the kernels (the present
code generation may keep it), so the declarations are read.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "turbins_gb300", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "pdl_wait(" in open(os.path.join(CSRC, f)).read())

# const tables formed when a context is created; kernels with reasons of their own
SETTLED = {
    "*": {"invd", "ainv", "st"},
    # r is the residual of the whole correction: the kernel that writes it has
    # ended before the first sweep, an ordinary launch, begins
    "k_helm_jac32v": {"r"},
    # the immersed rows' kernels work beside the stencil kernel ahead of them on
    # points that it does not write and end with their wait.  That kernel is an
    # ordinary launch, or has waited itself before it lets them start, so what
    # they read is complete.
    "k_ib_resid64": {"b", "x", "rf", "e0", "part"},
    "k_ib_jac32": {"r", "e", "en", "x"},
}


def kernels(path):
    """(name, parameters, body) of every __global__ function of a file"""
    src = open(path).read()
    src = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", src, flags=re.S))

    def close(at, pair):
        depth = 0
        for n in range(at, len(src)):
            depth += (src[n] == pair[0]) - (src[n] == pair[1])
            if depth == 0:
                return n
        raise AssertionError("unbalanced %s in %s" % (pair, path))

    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__)?", src):
        at = m.end()
        if src[at] == "(":
            at = close(at, "()") + 1
        op = src.index("(", at)
        cp = close(op, "()")
        ob = src.index("{", cp)
        yield src[at:op].strip(), src[op + 1:cp], src[ob:close(ob, "{}") + 1]


def unsettled(name, params):
    """arguments of a kernel whose loads may pass its wait"""
    bad = []
    for p in params.split(","):
        m = re.search(r"__restrict__\s*(\w+)", p)
        if m and not (("const" in p and m.group(1) in SETTLED["*"]) or m.group(1) in SETTLED.get(name, ())):
            bad.append(m.group(1))
    return bad


def test_the_reader_finds_a_planted_mistake(tmp_path):
    f = tmp_path / "k.cu"
    f.write_text("template <int G>\n__global__ void __launch_bounds__(256, G ? 4 : 2) k_a(L l, const double *__restrict__ p, const\n"
                 " float *__restrict__ invd, double *q) // pdl\n{ pdl_wait(); { q[0] = p[0]; } }\n"
                 "__global__ void k_b(const double *__restrict__ p) { /* pdl_wait */ }\n")
    ks = list(kernels(str(f)))
    assert [k[0] for k in ks] == ["k_a", "k_b"]
    assert unsettled(*ks[0][:2]) == ["p"]
    assert "pdl_wait" in ks[0][2] and "pdl_wait" not in ks[1][2]


@pytest.mark.parametrize("name", FILES)
def test_no_restrict_on_what_the_kernel_ahead_writes(name):
    early = [k for k in kernels(os.path.join(CSRC, name)) if "pdl_wait" in k[2]]
    assert early
    assert {k[0]: unsettled(k[0], k[1]) for k in early if unsettled(k[0], k[1])} == {}


def test_every_early_launch_follows_the_switch():
    """TURB_KV_PDL off means plain stream order for every kernel (a race is
    looked for that way): the launch attribute is set in one helper and the two
    cluster launches, each under a flag, and every call hands a flag on."""
    src = {f: open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))}
    where = {f: s.count("cudaLaunchAttributeProgrammaticStreamSerialization") for f, s in src.items()}
    assert {f: n for f, n in where.items() if n} == {"turb_internal.cuh": 1, "k_mg.cu": 1, "k_mglow.cu": 1}
    assert "cfg.numAttrs = early ? 1 : 0;" in src["turb_internal.cuh"]
    assert "cfg.numAttrs = H.pdl ? 2 : 1;" in src["k_mg.cu"]
    assert re.search(r"if \(pdl\) \{\s*at\[n\]\.id = cudaLaunchAttributeProgrammaticStreamSerialization", src["k_mglow.cu"])
    flags = [m.group(1) for s in src.values() for m in re.finditer(r"\b(?:launch_early|launch_k|net_launch|launch_pairs)\(([^,]+),", s)]
    assert set(flags) <= {"pdl", "early", "H.pdl", "n->pdl", "int early", "int pdl"} and len(flags) > 40


def test_every_kernel_launched_early_waits():
    """a kernel launched with the attribute that never waited would run beside
    the one ahead of it"""
    untriggered, n = [], 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        path = os.path.join(CSRC, f)
        body = {k[0]: k[2] for k in kernels(path)}
        src = open(path).read()
        launched = set(re.findall(r"\b(?:launch_early|launch_k|net_launch|launch_pairs)\([^,]+,\s*(k_\w+)", src))
        launched |= set(re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(k_\w+)", src))
        launched |= {"k_helm_jac32v"} & set(body)   # launched through a variable
        assert all("pdl_wait()" in body[k] for k in launched), f
        untriggered += [k for k in sorted(launched) if "pdl_trigger()" not in body[k]]
        n += len(launched)
    assert n > 25
    # the immersed rows' kernels let nothing start before they end
    assert sorted(untriggered) == ["k_ib_jac32", "k_ib_resid64"]
