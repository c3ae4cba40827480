"""`weight_cast_scope` and `wgrad_in_place` belong to the thread that entered them."""
import threading

import pytest
import torch

import ulm_ops


def _in_turn(a, b):
    """Runs the steps of two generators alternately, each in a thread of its own; returns what each yielded."""
    gens, out, errors, over = {'a': a, 'b': b}, {'a': [], 'b': []}, [], set()
    gates = {'a': threading.Semaphore(1), 'b': threading.Semaphore(0)}

    def run(me, other):
        while len(over) < 2:
            gates[me].acquire()
            try:
                if me not in over:
                    out[me].append(next(gens[me]))
            except StopIteration:
                over.add(me)
            except Exception as e:                        # noqa: BLE001 - raised by the test's own thread
                errors.append(e)
                over.add(me)
            gates[other].release()

    threads = [threading.Thread(target=run, args=x, daemon=True) for x in (('a', 'b'), ('b', 'a'))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=60)
    if errors:
        raise errors[0]
    return out


def test_interleaved_cast_scopes_do_not_share_copies():
    x = torch.ones(1, 8, dtype=torch.bfloat16)
    w = torch.nn.Parameter(torch.ones(8, 8))

    def trainer():
        with ulm_ops.weight_cast_scope():
            ulm_ops.linear(x, w)
            yield
        with torch.no_grad():
            w.fill_(2.0)                                  # an optimiser step
        yield
        with ulm_ops.weight_cast_scope():
            yield
            yield float(ulm_ops.linear(x, w).detach()[0, 0])

    def scorer():
        with ulm_ops.weight_cast_scope():
            yield
            yield
        yield                                             # left between the trainer's entering and using its second scope

    assert _in_turn(trainer(), scorer())['a'][-1] == 16.0
    assert float(ulm_ops.linear(x, w).detach()[0, 0]) == 16.0


def test_a_scope_does_not_keep_copies_of_weights_that_are_computed():
    x = torch.ones(1, 8, dtype=torch.bfloat16)
    base = torch.nn.Parameter(torch.ones(8, 8))
    with ulm_ops.weight_cast_scope():
        for k in (1.0, 2.0):
            w = base * k
            y = ulm_ops.linear(x, w)
            y.sum().backward()
            assert float(y.detach()[0, 0]) == 8 * k
    assert torch.equal(base.grad, torch.full((8, 8), 3.0))


@pytest.mark.gpu
def test_in_place_weight_gradients_stay_in_their_thread():
    x = torch.randn(16, 64, device='cuda', dtype=torch.float16)
    w = torch.nn.Parameter(torch.randn(64, 64, device='cuda'))
    w.grad = torch.zeros_like(w)

    def trainer():
        with ulm_ops.wgrad_in_place():
            yield
            yield

    def other():
        with torch.autocast('cuda', dtype=torch.float16):
            y = ulm_ops.linear(x, w)
        yield torch.autograd.grad(y.float().sum(), w)[0]
        yield

    got = _in_turn(trainer(), other())['b'][0]
    assert got is not None and not w.grad.any()


@pytest.mark.gpu
def test_a_copy_is_used_on_the_stream_that_made_it():
    x = torch.ones(4, 64, device='cuda', dtype=torch.float16)
    w = torch.nn.Parameter(torch.ones(64, 64, device='cuda'))
    side = torch.cuda.Stream()
    with torch.no_grad(), ulm_ops.weight_cast_scope(ulm_ops.weight_copies([w], torch.float16)):
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as main:
            ulm_ops.linear(x, w)
        with torch.cuda.stream(side), torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as other:
            y = ulm_ops.linear(x, w)
    torch.cuda.synchronize()
    casts = [sum(e.count for e in p.key_averages() if e.key == 'aten::_to_copy') for p in (main, other)]
    assert casts == [0, 1] and bool((y == 64).all())


def test_the_cpu_step_needs_no_build(monkeypatch):
    import _native as N
    import ulm_dp

    def missing():
        raise RuntimeError('not built')

    for name in ('ext', 'lib', '_load_ext', '_load'):
        monkeypatch.setattr(N, name, missing)
    monkeypatch.setattr(N, '_ext', None)
    monkeypatch.setattr(N, '_ext_error', None, raising=False)

    class Model(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.embedding, self.head = torch.nn.Embedding(11, 8), torch.nn.Linear(8, 11, bias=False)

        def compute_loss(self, ids, ignore_index=0, chunk_rows=0, denominator=None):
            z = ulm_ops.linear(self.embedding(ids[:, :-1]), self.head.weight)
            return torch.nn.functional.cross_entropy(z.reshape(-1, 11), ids[:, 1:].reshape(-1), ignore_index=ignore_index, reduction='sum') / denominator

    def post(flat, inv_scale, out):
        flat.mul_(inv_scale)
        out[0] += flat.square().sum()

    torch.manual_seed(0)
    model = Model()
    before = model.head.weight.detach().clone()
    cost = ulm_dp.CostModel.for_model(100.0, 8, 1, False)
    step = ulm_dp.DataParallelStep(model, torch.optim.SGD(model.parameters(), 0.1), samples_per_step=4, grad_post=post, cost=cost)
    loss, norm, skipped = step.step([torch.randint(1, 11, (4, 6))])
    assert float(loss) > 0 and float(norm) > 0 and not skipped and not torch.equal(before, model.head.weight)


@pytest.mark.gpu
def test_the_copies_outlive_the_work_of_every_stream_that_used_them():
    w = torch.nn.Parameter(torch.ones(1024, 1024, device='cuda'))
    x = torch.ones(4, 1024, device='cuda', dtype=torch.float16)
    copies = ulm_ops.weight_copies([w], torch.float16)
    torch.cuda.synchronize()
    side, where = torch.cuda.Stream(), copies.views[0].data_ptr()
    with torch.no_grad(), torch.cuda.stream(side):
        torch.cuda._sleep(200_000_000)                    # about 0.1 s of clock cycles, in front of the copies' use
        with ulm_ops.weight_cast_scope(copies):
            y = ulm_ops.linear(x, w)
    del copies
    other = torch.full((1024, 1024), 2.0, device='cuda', dtype=torch.float16)
    assert other.data_ptr() != where
    torch.cuda.synchronize()
    assert bool((y == 1024).all())
