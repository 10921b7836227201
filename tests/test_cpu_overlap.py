"""Passes that may overlap their predecessor (launch_pass) are resident while
it still writes; the read-only data path is for data that does not change in
a kernel's lifetime, so they must not read a predecessor's output through it.
No wrong value shows on a GPU (the loads come after the wait), so the sources
are checked: no const __restrict__ pointer among the parameters of such a
pass, and no __ldg, but for the twiddle tables, the kernel octant and the
batch's tables."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "1_b200", "csrc")
# written before any pass that reads them is launched
CONSTANT = {"tw", "twP", "g", "starts"}


def sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        s = open(f).read()
        out[os.path.basename(f)] = re.sub(r"//[^\n]*", "", s)
    return out


def passes(src):
    """name -> (parameters, body) of every function that waits as a pass does."""
    found = {}
    for s in src.values():
        for m in re.finditer(r"\b(\w+)\(([^(){};]*)\)\s*\{", s):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(s[i], 0)
                i += 1
            if "pass_wait();" in s[m.end():i]:
                found[m.group(1)] = (m.group(2), s[m.end():i])
    return found


def test_passes_read_their_input_by_plain_loads():
    src = sources()
    fs = passes(src)
    wrap = {k: m.group(1) for k in ("k_zr2c_fx", "k_col_fx") for s in src.values()
            for m in re.finditer(r"\b%s\(([^(){};]*)\)\s*\{" % k, s)}
    assert set(wrap) == {"k_zr2c_fx", "k_col_fx"}
    for name, par in [(k, v[0]) for k, v in fs.items()] + list(wrap.items()):
        for p in par.split(","):
            if "__restrict__" in p:
                assert p.split()[-1] in CONSTANT, (name, p)
    for name, (_, body) in fs.items():
        for a in re.findall(r"__ldg\(([^;]*)", body):
            assert re.match(r"&?(z\.)?(tw|twP)\b", a), (name, a)
    # and the scan has found them all
    assert {"col_body", "conv_body", "conv_wide_body", "zr2c_body", "k_zc2r_fx", "zinv_body", "k_col_mix", "k_conv_mix",
            "k_zr2c_mix", "k_zc2r_mix", "k_zinv_mix"} == set(fs)


def test_only_passes_are_launched_as_such():
    """Every kernel given to launch_pass waits, itself or in its body function."""
    src = sources()
    fs = passes(src)
    names = set()
    for f, s in src.items():
        for m in re.finditer(r"launch_pass\(\s*(?:mix::)?(\w+)", s):
            if m.group(1) not in ("void", "kern"):
                names.add(m.group(1))
        if "launch_pass(kern" in s:
            names |= set(re.findall(r"go\((?:mix::)?(k_\w+)", s))
    assert len(names) >= 9
    for k in names:
        body = next(s[m.end():m.end() + 400] for s in src.values() for m in re.finditer(r"\b%s\([^(){};]*\)\s*\{" % k, s))
        calls = set(re.findall(r"\b(\w+)(?:<[^;{}]*?>)?\(", body))
        assert k in fs or calls & (set(fs) | {"conv_block"}), k
