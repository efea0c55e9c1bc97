"""Kernels that begin before the ones ahead of them have ended (csrc/seq_launch.cuh): what an earlier kernel writes must not be read
through the read-only path or through `__restrict__` parameters, which the compiler may move across the wait.  Read from the sources,
since a wrong value would depend on timing."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "kuiperllama_b200" / "csrc"
WEIGHTS = {"w", "bias", "qnorm_w", "knorm_w", "q_norm_w", "kv_norm_w", "sink", "w_uk", "w_uv", "decay", "gate_up", "down"}
WEIGHT_POINTERS = WEIGHTS | {"wr", "wg", "wu", "a.in_w", "a.out_w", "a.mix", "a.rope_freq"}


def body(text, start):
    depth, i = 1, start
    while depth:
        depth += (text[i] == "{") - (text[i] == "}")
        i += 1
    return text[start:i]


def early_kernels():
    out = []
    for path in sorted(CSRC.glob("seq_*.cu*")):
        text = path.read_text()
        for m in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\(([^{]*)\)\s*\{", text):
            code = body(text, m.end())
            if "after_previous()" in code:
                out.append((m.group(1), m.group(2), code))
    return out


KERNELS = early_kernels()


def test_kernels_were_found():
    assert len(KERNELS) >= 18
    assert {"rows_kernel", "qk_turn_kernel", "attention_kernel", "umma_split_kernel", "streams_kernel"} <= {k[0] for k in KERNELS}


@pytest.mark.parametrize("name,parameters,code", KERNELS, ids=[k[0] for k in KERNELS])
def test_only_weights_take_the_read_only_path(name, parameters, code):
    assert set(re.findall(r"__restrict__ (\w+)", parameters)) <= WEIGHTS
    assert "__restrict__" not in code
    read_only = r"(?:__ldg|Vec16<AT>::load_stream|Wide<AT>::template load<\w+>)\((?:reinterpret_cast<[^>]*>\()?([\w.]+)"
    assert set(re.findall(read_only, code)) <= WEIGHT_POINTERS
    assert "ld.global.nc" not in code


# what a kernel reads ahead of its wait: weights, and what was complete before the step's first kernel began
EARLY = {"rows_kernel": {"w"}, "rows_gated_kernel": {"w"}, "umma_split_kernel": {"map_w", "map_w2", "p"},
         "umma_f32_kernel": {"map_w", "map_w2", "p"}, "qk_turn_kernel": {"rope", "tok_pos"},
         "attention_rows_mma_kernel": {"ent_first", "ent_count", "ent_seq", "ent_pos0", "kv"}}


@pytest.mark.parametrize("name,parameters,code", KERNELS, ids=[k[0] for k in KERNELS])
def test_reads_ahead_of_the_wait(name, parameters, code):
    # up to the first wait that is not a row tile's without rows; whether a pointer is there is no access
    before = re.sub(r"if \(r0 >= n_rows\) \{\s*after_previous\(\);\s*return;\s*\}", "", code).split("after_previous()")[0]
    before = re.sub(r"\w+ != nullptr", "", before)
    memory = [p.split()[-1].lstrip("*&") for p in parameters.split(",") if not re.match(r"\s*(?:const )?(?:int|float|bool|AttnShape) \w+$", p)]
    assert {p for p in memory if re.search(rf"\b{p}\b", before)} <= EARLY.get(name, set())


def test_keys_of_the_step_come_after_the_wait():
    code = next(c for n, _, c in KERNELS if n == "attention_rows_mma_kernel")
    before, after = code[:code.rindex("after_previous()")], code[code.rindex("after_previous()"):]
    assert re.findall(r"load_tile\(.*?, (\w+), (\w+)\);", before) == [("true", "false")]
    assert re.findall(r"load_tile\(.*?, (\w+), (\w+)\);", after) == [("false", "true"), ("true", "true")]
    # a key of this step is one from pos0 on; the guard comes ahead of the table
    assert re.search(r"if \(valid && kj >= pos0 \? !mine : !old\) return;.*\n.*table\[", before)


def test_the_first_kernel_of_a_step_is_an_ordinary_launch():
    assert "embed_kernel" not in {k[0] for k in KERNELS}
    assert "embed_kernel<AT><<<" in (CSRC / "seq_kernels.cu").read_text()


def test_rows_are_loaded_coherently():
    """Vec16::load, by which the products of few rows read their rows."""
    text = (CSRC / "seq_gemm.cu").read_text()
    loads = [body(text, m.end()) for m in re.finditer(r" load\(const \w+\* p, float\* f\) \{", text)]
    assert len(loads) == 2 and not any("__ldg" in x or ".nc" in x for x in loads)


def test_joining_splits_reads_plain_pointers():
    assert "__restrict__" not in (CSRC / "seq_merge.cuh").read_text()
