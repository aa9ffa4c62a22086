"""Kernels that come up while their predecessor in the stream still runs
(tc::after_predecessor) read nothing but a run's fixed profiles before they
have waited for it, and must not use read-only loads (__ldg, a const
__restrict__ parameter) for what that predecessor writes: such loads are
defined only for memory nobody writes while the kernel lives, and the
compiler may move them ahead of the wait.  No device run can show that they
are absent, so the sources are read."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geophysics_gb300", "csrc")
# written once, by the host, before the first launch of a run
PROFILES = re.compile(r"\s*g\.[ca][xyz][12]\b")
# an array inside the kernel's parameters
PARAMS = ("g.it[",)


def functions():
    """Device functions of every file: (file, name) -> (parameters, body)."""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        s = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__(?:global|device)__[^;{}=]*?\b(\w+)\s*\(", s):
            if m.group(1) in ("__launch_bounds__", "__align__"):
                m = re.compile(r"\b(k_\w+)\s*\(").search(s, m.end())
                if not m:
                    continue
            i, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(s[i], 0)
                i += 1
            params = s[m.end():i]
            if not re.match(r"\s*\{", s[i:]):
                continue
            b = i = s.index("{", i)
            depth = 0
            while True:
                depth += {"{": 1, "}": -1}.get(s[i], 0)
                i += 1
                if not depth:
                    break
            key = (f, m.group(1))
            old = out.get(key, ("", ""))   # overloads together
            out[key] = (old[0] + params, old[1] + s[b:i])
    return out


FUNCS = functions()
EARLY = [k for k, (_, body) in FUNCS.items() if re.search(r"after_predecessor\(\)", body) and k[1].startswith("k_")]


def reached(key):
    """The kernel's body and those of the helpers of its file that it calls."""
    todo, seen = [key], []
    while todo:
        k = todo.pop()
        seen.append(k)
        for name in set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\(", FUNCS[k][1])):
            if (k[0], name) in FUNCS and (k[0], name) not in seen + todo:
                todo.append((k[0], name))
    return seen


def test_early_kernels_are_found():
    assert {n for _, n in EARLY} >= {"k_fused3d", "k_tti3d_vel", "k_tti3d_stress", "k_snap_store", "k_snap_image",
                                     "k_inject3d", "k_ae_e12", "k_ae_d21", "k_ae_d1", "k_tc_gemm", "k_tc_walk",
                                     "k_tc_wgrad"}


def test_no_read_only_loads_in_early_kernels():
    bad = []
    for key in EARLY:
        if re.search(r"const\s+\w+\s*\*\s*__restrict__", FUNCS[key][0]):
            bad.append((key, "const __restrict__"))
        for k in reached(key):
            body = FUNCS[k][1]
            bad += [(key, k[1], "ld.global.nc")] if "ld.global.nc" in body else []
            bad += [(key, k[1], body[m.start():m.end() + 40]) for m in re.finditer(r"__ldg\(", body)
                    if not PROFILES.match(body[m.end():])]
    assert not bad, bad


def test_nothing_is_read_before_the_wait():
    bad = []
    for key in EARLY:
        head = FUNCS[key][1].split("after_predecessor()")[0]
        bad += [(key, m.group(0)) for m in re.finditer(r"\b(?:tma[23]\s*\(|row_copy\s*\(|[a-z]\.\w+\[)", head)
                if not PROFILES.match(m.group(0)) and m.group(0) not in PARAMS]
    assert not bad, bad
