"""A call's grid plan is reused by the next call of its direction with the same
key; what a caller asks of the plan (its direction, a forced kernel, a batch
plan's chunk length) belongs to the key, or one caller would get another's.
(Checked in the source.)"""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wsclean_b200", "csrc")


def test_key_holds_what_callers_ask():
    src = open(os.path.join(CSRC, "wsg_context.cu")).read()
    key = re.search(r"std::array<double, \d+> key\{(.*?)\};", src, re.S).group(1)
    plan = open(os.path.join(CSRC, "wsg_plan.cu")).read() + src
    asked = set(re.findall(r"\bgp\.(\w+) = [^;]*;", plan))
    for f in ("nx", "ny", "gridding", "force_W", "force_sigma", "batch"):
        assert f in asked, f
    for f in sorted(asked):
        assert re.search(r"\bgp\." + f + r"\b", key), f
