// aclsparseSpMV / aclsparseSpMM / aclsparseSpMVOp with their unchanging arguments in one struct (b200sp_packed.h).
#include "internal.h"
#include "b200sp_packed.h"

extern "C" {

aclsparseStatus_t b200spPackedSpMV(const b200spPackedCall *c, float alpha, float beta)
{
    return aclsparseSpMV(c->handle, (aclsparseOperation_t)c->opA, &alpha, static_cast<aclsparseConstSpMatDescr_t>(c->a),
                         static_cast<aclsparseConstDnVecDescr_t>(c->x), &beta, static_cast<aclsparseDnVecDescr_t>(c->out),
                         ACL_FLOAT, (aclsparseSpMVAlg_t)c->alg, c->buffer);
}

aclsparseStatus_t b200spPackedSpMM(const b200spPackedCall *c, float alpha, float beta)
{
    return aclsparseSpMM(c->handle, (aclsparseOperation_t)c->opA, (aclsparseOperation_t)c->opB, &alpha,
                         static_cast<aclsparseConstSpMatDescr_t>(c->a), static_cast<aclsparseConstDnMatDescr_t>(c->x), &beta,
                         static_cast<aclsparseDnMatDescr_t>(c->out), ACL_FLOAT, (aclsparseSpMMAlg_t)c->alg, c->buffer);
}

aclsparseStatus_t b200spPackedSpMVOp(const b200spPackedCall *c, float alpha, float beta)
{
    return aclsparseSpMVOp(c->handle, static_cast<aclsparseSpMVOpPlan_t>(const_cast<void *>(c->a)), &alpha, &beta,
                           static_cast<aclsparseConstDnVecDescr_t>(c->x), static_cast<aclsparseConstDnVecDescr_t>(c->y),
                           static_cast<aclsparseDnVecDescr_t>(c->out));
}

}  // extern "C"
