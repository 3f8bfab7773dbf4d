"""What every kernel source has to keep, read from the sources: no GPU and no compiler needed, and none could show it (a load that the compiler moves in front of a wait gives
the right number on most days)."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sllm_b200", "csrc")
SOURCES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# What no kernel of a step writes: matrices, gains, biases, tables, and constants of a layer.
CONSTANTS = set("W w table pair_table bias gain gain_a gain_b q_gain k_gain post_gain pre_gain ga gb conv_w inv_freq correction sink rel q_mul mix share into vec".split())
# What a kernel only writes.
RESULTS = set("out out_h out_hs out_a out_b q_out h dst C idx wts dense place tile_expert row_token k_cache v_cache pk_cache pv_cache cache partial rinv".split())
# Blocks in shared memory (chunked.cuh, delta_chunks.cu), and zero_rows' table, which its owner writes once.
ELSEWHERE = {("chunked.cuh", n) for n in ("A", "B", "dst")} | {("delta_chunks.cu", n) for n in ("m", "v", "lt", "col", "A0", "A1", "B")} | {("elementwise.cu", "long long rows")}


def code_of(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


@pytest.mark.parametrize("name", SOURCES)
def test_what_an_earlier_kernel_writes_is_loaded_behind_the_wait(name):
    """A kernel is set up while the one before it runs, and waits for it in `pdl_wait()`.  ``const __restrict__`` says that nobody writes there while the kernel runs, so the compiler may
    move the load in front of the wait: a pointer to what the step itself produces has no such qualifier."""
    wrong = []
    for const, kind, pointer in re.findall(r"(const\s+)?((?:long\s+)?[\w:]+)\s*\*\s*__restrict__\s+(\w+)", code_of(name)):
        if (name, pointer) in ELSEWHERE or (name, f"{kind} {pointer}") in ELSEWHERE:
            continue
        if pointer not in (CONSTANTS if const else RESULTS):
            wrong.append(pointer)
    assert not wrong, f"{name}: __restrict__ on {wrong}"


@pytest.mark.parametrize("name", SOURCES)
def test_read_only_loads_are_of_constants(name):
    """`__ldg` reads what nobody writes while the kernel runs, and the kernel runs while the one before it still writes (`__ldcg` is no more ordered behind the wait): both are for constants."""
    arguments = [code_of(name)[m.end():].lstrip() for m in re.finditer(r"__ldc?g\(", code_of(name))]
    constants = ("p.a_log", "p.skip", "p.a_bias", "p.dt_bias", "p.rel", "rel_h[", "bias", "tab ", "reinterpret_cast<const float4*>(bias", "reinterpret_cast<const float4*>(w ")
    assert not [a[:60] for a in arguments if not a.startswith(constants)]


@pytest.mark.parametrize("name", SOURCES)
def test_settings_of_a_kernel_are_made_on_every_device(name):
    """A kernel's limit of shared memory and its split of L1 lie with a device's copy of it: no flag or size of the whole process says that they have been set (`SharedLimit`; a bit a device)."""
    code = code_of(name)
    assert not re.findall(r"\bstatic (?:bool|int|size_t) \w+ =[^=(]*;", code)
    if name not in ("common.cuh", "linear_ws.cu", "gemm_f32.cu"):           # (gemm_f32.cu sets it at every launch)
        assert "cudaFuncSetAttribute" not in code


def test_the_rotary_epilogue_reads_positions_and_slots_behind_the_wait():
    """A slot read before the kernels that came earlier have finished would send keys and values to another request's page, without an error, a position turn them by another's angle."""
    code = code_of("linear_ws.cu")
    code = code[code.index("linear_ws_kernel("):]
    wait = code.index("pdl_wait();")
    early, late = code[:wait], code[wait:]
    assert "rope.slot_mapping" not in early and early.count("rope.positions") == 1 and "token_s[0][ahead_tok] = min(max(ws_position(rope.positions" in early
    assert "ws_copy4(&token_s[1][ahead_tok], rope.positions" in late and "ws_copy4(&token_s[2][ahead_tok], rope.slot_mapping" in late and "if (pos != token_s[0][tok])" in late
