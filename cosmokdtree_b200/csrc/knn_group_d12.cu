// knn_group_d12.cu -- the kNN kernel with a group of lanes per query, d = 1 and 2.
#include "ckd_knn_group.cuh"

namespace ckd {
CKD_KNN_GROUP(1)
CKD_KNN_GROUP(2)
}  // namespace ckd
