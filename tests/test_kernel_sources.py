"""Rules that the kernels' sources keep, checked by reading them.

A kernel that is launched with programmatic dependent launch is resident while the kernel in
front of it still runs, and reads that kernel's results after ``griddepcontrol.wait``. A pointer
parameter declared ``__restrict__`` promises the compiler that nothing else touches the data
during the kernel, which allows it to fetch the data (through the read-only path) ahead of the
wait. That happened once to the kernel that merges the attention splits. So in every kernel
that waits for its predecessor only weights, constants and the step's metadata, which are on
the device before the chain starts, may carry the qualifier."""

from __future__ import annotations

import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "llm-inference_b200" / "csrc" / "kernels"

# Parameters that hold weights, constants or step metadata: written before the chain of kernels
# starts, never by a kernel of the chain.
BEFORE_THE_CHAIN = {
    "W", "table", "weight", "bias", "inv_freq", "positions", "token_seq", "seq_kv_len", "block_table",
    # weights and constants of the post-norm blocks, the latent attention and the delta rule
    "scale", "mix", "coefficients", "norm_weight", "sink", "taps_w", "a_log", "dt_bias",
    # stream weights of the hyper-connections, blend factors, decay offset and bonus of the recurrent mixer with a bonus
    "mix_w", "out_w", "in_w", "mu", "w0", "u",
    # the step's per-request metadata; norm weights over all heads, weights of a pair of mixers, the pair table
    "seq_q_start", "seq_q_len", "seq_slot", "a_bias", "q_weight", "k_weight", "wa", "wb", "pairs",
    "blend",  # factors of the blend with the previous token's row
}


def global_kernels(text: str):
    """(name, parameter list, body) of every ``__global__`` function of a source file."""
    for match in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        start = match.end()
        depth, at = 1, start
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params = text[start : at - 1]
        brace = text.index("{", at)
        depth, end = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield match.group(1), params, text[brace:end]


def test_kernels_that_wait_for_their_predecessor_keep_restrict_for_what_precedes_the_chain():
    seen = 0
    for path in sorted(KERNELS.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for name, params, body in global_kernels(text):
            if "wait_for_predecessor" not in body:
                continue
            seen += 1
            for param in params.split(","):
                if "__restrict__" not in param:
                    continue
                pname = param.split()[-1]
                assert pname in BEFORE_THE_CHAIN, (
                    f"{path.name}: {name}({pname}) is __restrict__ in a kernel that runs beside its predecessor")
    assert seen >= 10  # the rule found the kernels it is about


def test_the_rule_reads_a_kernel_as_intended():
    sample = """
    template <typename T>
    __global__ void __launch_bounds__(128)
    demo_kernel(const T* __restrict__ weight, const T* __restrict__ x, int n) {
      wait_for_predecessor();
      if (n) { x[0]; }
    }
    """
    (name, params, body), = list(global_kernels(sample))
    assert name == "demo_kernel" and "wait_for_predecessor" in body
    restricted = [p.split()[-1] for p in params.split(",") if "__restrict__" in p]
    assert restricted == ["weight", "x"] and "x" not in BEFORE_THE_CHAIN


def test_limits_of_shared_memory_are_raised_on_every_device():
    """A flag that a process sets once leaves its second device with the first limit, and keeps a failure for good."""
    for path in sorted(KERNELS.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        assert not re.search(r"static\s+const\s+bool\s+\w+\s*=", text), path.name


def test_what_is_done_once_per_device(tmp_path):
    """The class behind those limits, against a device number and an action that the test sets."""
    import shutil
    import subprocess

    import pytest

    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no C++ compiler")
    found = re.search(r"constexpr int kMaxDevices = \d+;\nclass OncePerDevice \{.*?\n\};", (KERNELS / "common.cuh").read_text(), re.S)
    (tmp_path / "once.cpp").write_text(
        "#include <atomic>\n#include <cassert>\n"
        "enum { cudaSuccess = 0 };\nstatic int current = 0, refused = 0;\n"
        "static int cudaGetDevice(int* d) { *d = current; return refused; }\nstatic int cudaGetLastError() { return 0; }\n"
        + found.group(0) + "\n"
        "int main() {\n  OncePerDevice once;\n  int runs = 0, works = 0;\n  auto action = [&] { ++runs; return works != 0; };\n"
        "  assert(!once(action) && !once(action) && runs == 2);  // a failure is not kept\n"
        "  works = 1;\n  assert(once(action) && once(action) && runs == 3);\n"
        "  current = 1;\n  assert(once(action) && once(action) && runs == 4);\n"
        "  current = kMaxDevices;\n  assert(!once(action) && runs == 4);\n"
        "  current = 0, refused = 1;\n  assert(!once(action) && runs == 4);\n  return 0;\n}\n"
    )
    subprocess.run([compiler, "-std=c++17", "-o", str(tmp_path / "once"), str(tmp_path / "once.cpp")], check=True)
    subprocess.run([str(tmp_path / "once")], check=True)


def test_recurrences_that_walk_portions_are_launched_the_ordinary_way():
    """Resident early, their few long-lived blocks share the SMs that the kernel in front leaves first: 100 tokens of 24 heads of
    64 x 64 walked in 80 us instead of 30 once the kernel in front had become short."""
    for name, entry in (("delta_head", "b200_delta_head_recurrence"), ("delta_general", "b200_delta_general_recurrence"), ("wkv", "b200_wkv_recurrence")):
        text = (KERNELS / f"{name}.cu").read_text()
        body = text[text.index(f"B200_API int {entry}(") :]
        body = body[: body.index("\n}\n")]
        assert "const bool ordered = max_q_len > kStage;" in body and "launch_kernel_as(ordered, kernel" in body, entry
