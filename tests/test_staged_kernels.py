"""The kernels that wait for staged copies leave together when one does not
complete.  Their column barriers (named, of a fixed number of threads) wait for
every thread, so a thread may not return on the outcome of its own wait: the
source of every such kernel turns the outcome into a barrier's vote first.
(Checked in the source: no run makes a copy fail.)"""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _kernels():
    for path in sorted(glob.glob(os.path.join(ROOT, "wsclean_b200", "csrc", "*.cuh"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\([^{;]*\)\s*\{", src):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[i], 0)
                i += 1
            yield m.group(1), src[m.end():i]


def test_waits_are_voted_on():
    seen = []
    for name, body in _kernels():
        if "mbar_wait(" not in body:
            continue
        seen.append(name)
        # no branch on a thread's own wait ...
        assert not re.search(r"if\s*\(\s*!?\s*mbar_wait\(", body), name
        # ... and the kernel leaves early on a vote of the whole CTA only
        votes = len(re.findall(r"if \(__syncthreads_or\(", body))
        returns = len(re.findall(r"atomicOr\(err, 2\);\s*mbar_wait\([^)]*\);\s*return;", body))
        assert votes == returns >= 1 and body.count("atomicOr(err") == returns, name
    assert set(seen) >= {"k_ucol_bwd_tma", "k_ucol_fwd_bulk", "k_ucol_bwd_quad", "k_ucol_fwd_quad"}
