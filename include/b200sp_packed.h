/*
 * b200sp_packed.h -- compute calls whose unchanging arguments are packed once, for callers behind a foreign-function
 * interface.
 *
 * A product on a small matrix takes about as long as an interpreter needs to convert the ten or more arguments of
 * aclsparseSpMV / aclsparseSpMM / aclsparseSpMVOp.  A caller that repeats a product fills a b200spPackedCall once
 * and then passes its address and the two scalars.  The calls are the aclsparse ones in every other respect: the
 * handle's pointer mode must be HOST, computeType ACL_FLOAT.  The struct is only read.
 */
#ifndef B200SP_PACKED_H_
#define B200SP_PACKED_H_

#include "cann_ops_sparse.h"

#ifdef __cplusplus
extern "C" {
#endif

typedef struct b200spPackedCall {
    aclsparseHandle_t handle;
    const void *a;   /* matA, or the aclsparseSpMVOpPlan_t */
    const void *x;   /* vecX or matB */
    const void *y;   /* SpMVOp: vecY */
    void *out;       /* vecY, matC, or SpMVOp: vecZ */
    void *buffer;
    int opA, opB, alg;
} b200spPackedCall;

aclsparseStatus_t b200spPackedSpMV(const b200spPackedCall *call, float alpha, float beta);
aclsparseStatus_t b200spPackedSpMM(const b200spPackedCall *call, float alpha, float beta);
aclsparseStatus_t b200spPackedSpMVOp(const b200spPackedCall *call, float alpha, float beta);

#ifdef __cplusplus
}
#endif

#endif /* B200SP_PACKED_H_ */
