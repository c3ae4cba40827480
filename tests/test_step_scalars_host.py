"""What the step's small kernels take, decided on the host: nothing is launched here."""
import pytest
import torch

import ulm_model
import ulm_ops


def _reference(ids, labels, padded, ignore):
    n, L = ids.shape
    want = torch.full((n, L), ignore)
    want[:, :-1] = labels[:, 1:]
    return torch.cat([ids.reshape(-1).long(), torch.zeros(padded - n * L, dtype=torch.long)]), torch.cat([want.reshape(-1), torch.full((padded - n * L,), ignore)])


@pytest.mark.parametrize('dtype', [torch.int64, torch.int32])
@pytest.mark.parametrize('labels', ['same', 'one row'])
def test_token_targets_off_the_kernels_form(dtype, labels):
    ids = torch.randint(1, 99, (3, 5)).to(dtype)
    lab = ids if labels == 'same' else ids[:1].long()
    flat, target = ulm_ops.token_targets(ids, lab, 32, -7)
    want = _reference(ids, lab, 32, -7)
    assert torch.equal(flat.long(), want[0]) and torch.equal(target, want[1]) and target.dtype == torch.long


@pytest.mark.parametrize('labels', [torch.zeros(3, 4, dtype=torch.long), torch.zeros(2, 5, dtype=torch.long), torch.zeros(3, 5)])
def test_token_targets_refuses_labels_that_do_not_fit(labels):
    with pytest.raises((ValueError, RuntimeError)):
        ulm_ops.token_targets(torch.ones(3, 5, dtype=torch.long), labels, 32, 0)


def test_compute_loss_on_host_tensors_raises_and_launches_nothing():
    import _native as N
    model = ulm_model.DecoderOnlyTransformer(ulm_model.ModelConfig(vocab_size=64, d_model=64, n_layers=1, n_heads=1, d_ff=64, max_seq_len=32))
    before = N.lib().ulm_launch_count()
    with pytest.raises(ValueError):
        model.compute_loss(torch.ones(2, 8, dtype=torch.long))
    assert N.lib().ulm_launch_count() == before


@pytest.mark.parametrize('kept', [True, False])
@pytest.mark.parametrize('target', [torch.ones(4, dtype=torch.int32), torch.ones(3, dtype=torch.long), torch.ones(4, dtype=torch.long, device='meta')])
def test_cross_entropy_refuses_targets_its_kernels_cannot_read(target, kept, monkeypatch):
    monkeypatch.setattr(ulm_ops, 'KEEP_LOGITS_BYTES', ulm_ops.KEEP_LOGITS_BYTES if kept else 0)
    with pytest.raises(ValueError):
        ulm_ops.chunked_cross_entropy(torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(64, 64), target, denominator=1.0)


@pytest.mark.parametrize('flat,sumsq', [(torch.zeros(8), torch.zeros(1)), (torch.zeros(8, device='meta'), torch.zeros(1, device='meta')),
                                        (torch.zeros(8, dtype=torch.float16), torch.zeros(1))])
def test_grad_clip_refuses_what_its_kernel_cannot_read(flat, sumsq):
    with pytest.raises(ValueError):
        ulm_ops.grad_clip_(flat, sumsq, 1.0)
