"""Kernels launched before their predecessor ends (programmatic dependent
launch) read what earlier launches wrote through plain loads only.

Such a grid is resident while its predecessor still writes, so a vector is
not read-only for its lifetime: the read-only path (__ldg, a const
__restrict__ pointer) is only for what is written at set-up.  The sources are
read here, since the compiler's choice shows in no result that a test could
count on.
"""
import glob
import os
import re

from conftest import ROOT

# what is written at set-up and never again while a kernel may read it
SETUP = {
    "ia", "ja", "a", "ia0", "ja0", "a0",        # matrices
    "dj", "vi", "vtab", "edj", "evi", "split",  # packed, ELL and windowed forms
    "S",                                        # stencil masks
    "mu0", "muk",                               # polynomial coefficients
    "B", "bias", "mask",                        # network: weights, stored inputs
    "T",                                        # network: the caller's targets
}


def functions():
    """name -> list of source texts (signature and body) of every function."""
    out = {}
    for f in sorted(glob.glob(os.path.join(ROOT, "pevsl_b200", "csrc", "*.cu*"))):
        text = re.sub(r"/\*.*?\*/", " ", open(f).read(), flags=re.S)
        text = re.sub(r"//[^\n]*", " ", text)
        for m in re.finditer(r"__(?:global|device)__", text):
            i = text.find("{", m.end())
            semi = text.find(";", m.end())
            if i < 0 or 0 <= semi < i:
                continue  # a declaration
            head = text[m.start():i]
            head_flat = re.sub(r"__launch_bounds__\s*\([^)]*\)", " ", head)
            name = re.search(r"(\w+|operator\(\))\s*\(", head_flat)
            depth, j = 0, i
            while True:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
                if depth == 0:
                    break
            out.setdefault(name.group(1) if name else "", []).append((os.path.basename(f), text[m.start():j]))
    return out


def closure(funcs, text, seen):
    """the texts of all device functions that a body calls, directly or not"""
    for w in set(re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\s*\(", text)):
        if w in funcs and w not in seen and not w.startswith("k_"):
            seen.add(w)
            for _, t in funcs[w]:
                yield w, t
                yield from closure(funcs, t, seen)


def violations(name, text):
    bad = []
    for m in re.finditer(r"const\s+[\w:]+\s*\*\s*__restrict__\s*(\w+)", text):
        if m.group(1) not in SETUP:
            bad.append(f"{name}: const __restrict__ {m.group(1)}")
    for m in re.finditer(r"__ldg\(\s*(?:\([^()]*\)\s*)?(\w+)", text):
        if m.group(1) not in SETUP:
            bad.append(f"{name}: __ldg({m.group(1)}")
    return bad


def test_dependent_kernels_read_vectors_through_plain_loads():
    funcs = functions()
    kernels = {n: t for n, v in funcs.items() for _, t in v
               if "__global__" in t and "pdl_wait_then_release" in t}
    assert {"k_csr_stream", "k_cheb_stencil", "k_rows_stencil", "k_csr_window", "k_kpm_csr",
            "k_cheb_il_mid", "k_b_gemv_sub_nrm", "k_gemm_bf16", "k_mse"} <= set(kernels)
    bad = []
    for n, t in kernels.items():
        bad += violations(n, t)
        for w, d in closure(funcs, t, set()):
            bad += violations(f"{n} -> {w}", d)
    assert not bad, "\n".join(bad)


def test_every_dependent_launch_waits():
    """every kernel that a launch_pdl call names waits for its predecessor"""
    funcs = functions()
    for f in sorted(glob.glob(os.path.join(ROOT, "pevsl_b200", "csrc", "*.cu"))):
        text = open(f).read()
        for m in re.finditer(r"launch_pdl(?:_block)?\((k_\w+)", text):
            assert any("pdl_wait_then_release" in t for _, t in funcs[m.group(1)]), m.group(1)
