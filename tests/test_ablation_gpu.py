"""The benchmark's stand-ins for the kernels of a decode step: each takes away the launches that its name says, whichever form the step's
attention takes."""
import pytest
import torch

import bench
import rocmforge_b200 as rf
from helpers import TINY_D, write_tiny
from rocmforge_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim,batch,formed", [
    (16, 2, 64, 3, True), (8, 2, 128, 3, True),
    (16, 16, 128, 16, False)])                            # 256 (sequence, kv head) pairs of 128: the writer and the attention
def test_stand_ins_take_a_kernels_launches_away(tmp_path, heads, kv_heads, head_dim, batch, formed):
    L = 2
    write_tiny(dict(TINY_D, num_hidden_layers=L, hidden_size=1024, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim,
                    intermediate_size=1536), str(tmp_path), "bfloat16")
    model = rf.LLM(str(tmp_path), dtype="bfloat16").model
    cache = model.new_cache(max_tokens=batch * 128, max_slots=batch)
    slots = [cache.alloc_slot() for _ in range(batch)]

    def launches():
        before = kernels.launch_count()
        model.step(cache, [rf.StepRequest(s, [1], [0]) for s in slots])
        torch.cuda.synchronize()
        return kernels.launch_count() - before

    whole = launches()
    gone = {}
    for name, patches in bench.ablation_cases(model.config, model.device):
        with pytest.MonkeyPatch.context() as m:
            for module, attribute, stand_in in patches:
                m.setattr(module, attribute, stand_in)
            gone[name.split(" (")[0]] = whole - launches()
    assert launches() == whole
    assert gone == {"norm kernels": 2 * L + 1, "rotation + cache write": 0 if formed else L, "attention": L, "q|k|v product": L, "o product": L,
                    "gate/up product": L, "down product": L, "output matrix": 1, "all products": 4 * L + 1}
    kernels.tensor_core.check_status(model.device)
