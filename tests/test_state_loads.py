"""Step kernels start by programmatic dependent launch: one may be resident
while the kernel that writes its inputs still runs. A load through the
non-coherent path (__ldg, or a const __restrict__ kernel parameter, which lets
the compiler choose it) promises data nothing writes while the kernel lives,
and may be moved above the wait for the earlier kernel. So step kernels take
only the constant tables that way, never the model's state."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "web-exoplasim_b200", "csrc")
# Set-up kernels and the allocation-free sums are launched the ordinary way.
NOT_STEP = {"setup_device.cu", "noalloc.cu"}
# Tables no kernel of a step writes: the planets' constants and level tables,
# the DFT, twiddle and Legendre tables.
TABLES = {"pcr", "tabr", "tab", "twg", "qi", "qj", "qu", "qv", "qa", "qb", "bm1"}


def step_sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".h")) and name not in NOT_STEP:
            text = open(os.path.join(CSRC, name)).read()
            yield name, re.sub(r"//[^\n]*", "", text)


def test_read_only_loads_take_tables_alone():
    bad = []
    for name, text in step_sources():
        for m in re.finditer(r"(?:__ldg|__ldlu|ld\.global\.nc)\s*\(([^;]*)", text):
            names = set(re.findall(r"[A-Za-z_]\w*", re.sub(r"reinterpret_cast<[^>]*>", "", m.group(1))))
            if not names & TABLES:
                bad.append((name, m.group(0)[:60]))
    assert not bad, bad


def test_kernels_take_state_through_plain_pointers():
    bad = []
    for name, text in step_sources():
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\s*\(([^{;]*?)\)\s*\{", text):
            for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", m.group(2)):
                if p not in TABLES:
                    bad.append((name, m.group(1), p))
    assert not bad, bad
