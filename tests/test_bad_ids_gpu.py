"""Ids outside their tables: the kernels read nothing there, add nothing to any gradient and say so under the lookup's own name, at the step
itself where its results are fetched and otherwise at the next call or when the session closes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_pair_lookup_reads_zeros_and_reports():
    from autodist_b200.ops import functional as Fn
    tables = [torch.ones(k, 24, device="cuda").requires_grad_(True) for k in (6, 4)]
    for t in tables:
        t.grad, t._direct_grad = torch.zeros_like(t), True
    users, items = (torch.tensor(v, device="cuda") for v in ([0, 6, 2, -1, 5], [1, 1, 4, 2, 3]))
    gmf, x = Fn.pair_lookup(*tables, users, items, 8)
    torch.autograd.backward([gmf, x], [torch.ones_like(gmf), torch.ones_like(x)])
    with pytest.raises(RuntimeError, match="user, item"):
        Fn.check_errors()
    Fn.check_errors()                                                            # reported once
    good_u, good_i = torch.tensor([1., 0, 1, 0, 1], device="cuda"), torch.tensor([1., 1, 0, 1, 1], device="cuda")
    assert torch.equal(gmf, (good_u * good_i)[:, None].expand(5, 8))
    assert torch.equal(x.float(), torch.cat([good_u[:, None].expand(5, 16), good_i[:, None].expand(5, 16)], 1))
    assert torch.equal(tables[0].grad[:, 8:].sum(1), torch.tensor([16., 0, 16, 0, 0, 16], device="cuda"))
    assert torch.equal(tables[1].grad[:, 8:].sum(1), torch.tensor([0., 32, 16, 16], device="cuda"))


def test_sampled_softmax_reports():
    from autodist_b200.ops import functional as Fn
    raw, dot = torch.zeros(3, 8, device="cuda").bfloat16(), torch.zeros(3, device="cuda").bfloat16()
    bias = torch.zeros(9, device="cuda").requires_grad_(True)
    neg, own = torch.arange(8, device="cuda"), torch.tensor([1, 9, 2], device="cuda")
    for n, t in ((neg, own), (neg - 1, own.clamp(max=8))):
        Fn.sampled_softmax_of(raw, dot, bias, n, t, 8).backward()
        with pytest.raises(RuntimeError, match="outside its vocabulary"):
            Fn.check_errors()
    Fn.sampled_softmax_of(raw, dot, bias, neg, own, 8)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="outside its vocabulary"):            # the next call says it, without a check in between
        Fn.sampled_softmax_of(raw, dot, bias, neg, neg[:3], 8)
    Fn.check_errors()


@pytest.mark.parametrize("steps_before", [0, 4])
def test_a_session_raises_at_the_step(steps_before):
    """Eager steps and replayed ones."""
    from autodist_b200 import AutoDist
    from autodist_b200.autodist import _reset_default_autodist
    from autodist_b200.models.ncf import NeuMF, NeuMFConfig
    from autodist_b200.resource_spec import ResourceSpec
    from autodist_b200.strategy import AllReduce
    _reset_default_autodist()
    autodist = AutoDist(resource_spec=ResourceSpec.local(num_gpus=1), strategy_builder=AllReduce(chunk_size=64))
    c = NeuMFConfig.tiny(dense_gradient=True)
    good = {"users": torch.arange(16) % c.num_users, "items": torch.arange(16) % c.num_items, "labels": torch.zeros(16)}
    bad = dict(good, users=good["users"].clone().index_fill_(0, torch.tensor([3]), c.num_users))
    with autodist.scope():
        model = NeuMF(c)
        holders = {k: autodist.placeholder((None,), v.dtype, name=k) for k, v in good.items()}
        loss = model(**holders)
        train_op = torch.optim.Adam(model.parameters(), lr=1e-3).minimize(loss)
        session = autodist.create_distributed_session()

    def feed(batch):
        return {holders[k]: v for k, v in batch.items()}
    for _ in range(steps_before):
        session.run([loss, train_op], feed(good))
    with pytest.raises(RuntimeError, match="user, item"):
        session.run([loss, train_op], feed(bad))
    session.run([loss, train_op], feed(good))
    with pytest.raises(RuntimeError, match="user, item"):                        # nothing fetched: seen at the latest when the session closes
        session.run(train_op, feed(bad))
        session.close()
