"""Which arguments the ops take and which they refuse; refusals are decided on the host, before any launch."""
import pytest
import torch

import ulm_infer


@pytest.mark.parametrize('half', ['cos', 'sin'])
def test_causal_attention_wants_both_tables_or_none(half):
    with pytest.raises(ValueError, match='given together'):
        ulm_infer.causal_attention(torch.zeros(1, 4, 192, dtype=torch.float16), 1, **{half: torch.zeros(4, 64)})
