// Generated by gen_fastmath_tables.py (mpmath, 200-bit) - do not edit.
#pragma once

// 2^(j/512) 2^62, j = 0..511
#define FM_EXP_TABLE_INIT { \
  0x4000000000000000ull, \
  0x4016321b687027a8ull, \
  0x402c6be96af2fb58ull, \
  0x4042ad6cb2f445c2ull, \
  0x4058f6a7ecccd5b6ull, \
  0x406f479dc5c2d058ull, \
  0x4085a050ec0a036aull, \
  0x409c00c40ec437beull, \
  0x40b268f9de0183baull, \
  0x40c8d8f50ac09dffull, \
  0x40df50b846ef302bull, \
  0x40f5d046456a29b8ull, \
  0x410c57a1b9fe12f6ull, \
  0x4122e6cd59676024ull, \
  0x41397dcbd952c4a6ull, \
  0x41501c9ff05d8654ull, \
  0x4166c34c5615d0ecull, \
  0x417d71d3c2fb0999ull, \
  0x41942838f07e22a3ull, \
  0x41aae67e9901ef2dull, \
  0x41c1aca777db771bull, \
  0x41d87ab649524b14ull, \
  0x41ef50adcaa0d899ull, \
  0x42062e90b9f4be46ull, \
  0x421d1461d66f2023ull, \
  0x42340223e024fc1eull, \
  0x424af7d9981f7e98ull, \
  0x4261f585c05c5718ull, \
  0x4278fb2b1bce0d15ull, \
  0x429008cc6e5c54e0ull, \
  0x42a71e6c7ce464afull, \
  0x42be3c0e0d3949bbull, \
  0x42d561b3e6243d8aull, \
  0x42ec8f60cf64fb4aull, \
  0x4303c51791b21550ull, \
  0x431b02daf6b94ab1ull, \
  0x433248adc91fdd02ull, \
  0x43499692d482e625ull, \
  0x4360ec8ce577ae44ull, \
  0x43784a9ec98c01e2ull, \
  0x438fb0cb4f468808ull, \
  0x43a71f1546271899ull, \
  0x43be957f7ea712b6ull, \
  0x43d6140cca39b350ull, \
  0x43ed9abffb4c6bc9ull, \
  0x4405299be54738beull, \
  0x441cc0a35c8cf8eaull, \
  0x44345fd9367bc428ull, \
  0x444c0740496d4294ull, \
  0x4463b6db6cb703c6ull, \
  0x447b6ead78aad636ull, \
  0x44932eb946971eafull, \
  0x44aaf701b0c72feeull, \
  0x44c2c7899283a259ull, \
  0x44daa053c812abd2ull, \
  0x44f281632eb877afull, \
  0x450a6abaa4b77ecdull, \
  0x45225c5d0950dfc0ull, \
  0x453a564d3cc4b723ull, \
  0x4552588e2052780cull, \
  0x456a632296394492ull, \
  0x4582760d81b8467full, \
  0x459a9151c70f0819ull, \
  0x45b2b4f24b7dcd0cull, \
  0x45cae0f1f545eb73ull, \
  0x45e31553abaa2501ull, \
  0x45fb521a56ef0042ull, \
  0x46139748e05b220aull, \
  0x462be4e23237a6efull, \
  0x46443ae937d07cf5ull, \
  0x465c9960dd74bd4bull, \
  0x4675004c10770630ull, \
  0x468d6fadbf2dd4f3ull, \
  0x46a5e788d8f3e012ull, \
  0x46be67e04e28717cull, \
  0x46d6f0b7102fc0ecull, \
  0x46ef821011734e6bull, \
  0x47081bee45623ceaull, \
  0x4720be54a071ad01ull, \
  0x47396946181d17caull, \
  0x47521cc5a2e6a9e0ull, \
  0x476ad8d638579e75ull, \
  0x47839d7ad1009a90ull, \
  0x479c6ab6667a086aull, \
  0x47b5408bf36472e2ull, \
  0x47ce1efe7368e11eull, \
  0x47e70610e3393241ull, \
  0x47fff5c640907943ull, \
  0x4818ee218a3358eeull, \
  0x4831ef25bff05ff7ull, \
  0x484af8d5e2a06536ull, \
  0x48640b34f426e3fcull, \
  0x487d2645f7725895ull, \
  0x48964a0bf07c9cd9ull, \
  0x48af7689e44b44eaull, \
  0x48c8abc2d8effc0aull, \
  0x48e1e9b9d588e19bull, \
  0x48fb3071e240e632ull, \
  0x49147fee085028d6ull, \
  0x492dd83151fc545aull, \
  0x4947393eca98fcd6ull, \
  0x4960a3197e87fd44ull, \
  0x497a15c47b39d53eull, \
  0x49939142cf2e06d6ull, \
  0x49ad159789f37496ull, \
  0x49c6a2c5bc28bf9eull, \
  0x49e038d0777ca5e0ull, \
  0x49f9d7baceae6083ull, \
  0x4a137f87d58e025bull, \
  0x4a2d303aa0fcd694ull, \
  0x4a46e9d646edbf6aull, \
  0x4a60ac5dde65950full, \
  0x4a7a77d47f7b84b1ull, \
  0x4a944c3d43596f96ull, \
  0x4aae299b443c4a6bull, \
  0x4ac80ff19d747ca0ull, \
  0x4ae1ff436b663ff7ull, \
  0x4afbf793cb8a002aull, \
  0x4b15f8e5dc6cbab0ull, \
  0x4b30033cbdb05eaeull, \
  0x4b4a169b900c2d00ull, \
  0x4b643305754d1866ull, \
  0x4b7e587d905625d1ull, \
  0x4b9887070520ccd9ull, \
  0x4bb2bea4f8bd5847ull, \
  0x4bccff5a915346ccull, \
  0x4be7492af621abd6ull, \
  0x4c019c194f7f9081ull, \
  0x4c1bf828c6dc54b8ull, \
  0x4c365d5c86c01063ull, \
  0x4c50cbb7bacbf4cbull, \
  0x4c6b433d8fbaae12ull, \
  0x4c85c3f13360c4d5ull, \
  0x4ca04dd5d4acffe8ull, \
  0x4cbae0eea3a8c63cull, \
  0x4cd57d3ed17880e2ull, \
  0x4cf022c9905bfd32ull, \
  0x4d0ad19213aecf14ull, \
  0x4d25899b8fe8b365ull, \
  0x4d404ae93a9df28dull, \
  0x4d5b157e4a7fc325ull, \
  0x4d75e95df75caccdull, \
  0x4d90c68b7a20eb1eull, \
  0x4dabad0a0cd6d0bfull, \
  0x4dc69cdceaa72a9cull, \
  0x4de196074fd9a344ull, \
  0x4dfc988c79d52661ull, \
  0x4e17a46fa720445aull, \
  0x4e32b9b417619617ull, \
  0x4e4dd85d0b6020dfull, \
  0x4e69006dc503ba65ull, \
  0x4e8431e987556cf1ull, \
  0x4e9f6cd3967fdba8ull, \
  0x4ebab12f37cfa702ull, \
  0x4ed5feffb1b3d155ull, \
  0x4ef156484bbe2390ull, \
  0x4f0cb70c4ea39210ull, \
  0x4f28214f043ca19bull, \
  0x4f439513b785cc80ull, \
  0x4f5f125db49fe7d3ull, \
  0x4f7a993048d088d7ull, \
  0x4f96298ec2826a82ull, \
  0x4fb1c37c7145d328ull, \
  0x4fcd66fca5d0fa4aull, \
  0x4fe91412b2006e83ull, \
  0x5004cac1e8d77ba2ull, \
  0x50208b0d9e8090dfull, \
  0x503c54f9284da734ull, \
  0x50582887dcb8a7e1ull, \
  0x507405bd1363d309ull, \
  0x508fec9c251a267cull, \
  0x50abdd286bcfc49dull, \
  0x50c7d76542a25b72ull, \
  0x50e3db5605d98bd4ull, \
  0x50ffe8fe12e750c4ull, \
  0x511c0060c86866e2ull, \
  0x513821818624b40cull, \
  0x51544c63ad0faf1dull, \
  0x5170810a9f48c7cfull, \
  0x518cbf79c01bcecaull, \
  0x51a907b474015dc9ull, \
  0x51c559be209f3ff0ull, \
  0x51e1b59a2cc8da3eull, \
  0x51fe1b4c007f9426ull, \
  0x521a8ad704f3404full, \
  0x5237043ea4828572ull, \
  0x525387864abb4762ull, \
  0x527014b1645b1038ull, \
  0x528cabc35f4f799dull, \
  0x52a94cbfaab69642ull, \
  0x52c5f7a9b6df5b77ull, \
  0x52e2ac84f54a0ae6ull, \
  0x52ff6b54d8a89c75ull, \
  0x531c341cd4df284eull, \
  0x533906e05f045106ull, \
  0x5355e3a2ed61adf0ull, \
  0x5372ca67f774358full, \
  0x538fbb32f5eca831ull, \
  0x53acb60762affaaeull, \
  0x53c9bae8b8d7c147ull, \
  0x53e6c9da74b29ab5ull, \
  0x5403e2e013c49b51ull, \
  0x542105fd14c7b869ull, \
  0x543e3334f7ac33b8ull, \
  0x545b6a8b3d990704ull, \
  0x5478ac0368ec4fdfull, \
  0x5495f7a0fd3bbb8eull, \
  0x54b34d677f54f319ull, \
  0x54d0ad5a753e077cull, \
  0x54ee177d6635de01ull, \
  0x550b8bd3dab49cbdull, \
  0x55290a615c6c1730ull, \
  0x5546932976483b15ull, \
  0x5564262fb46f7d4cull, \
  0x5581c377a44346f0ull, \
  0x559f6b04d4606293ull, \
  0x55bd1cdad49f699cull, \
  0x55dad8fd361531cdull, \
  0x55f89f6f8b133af4ull, \
  0x5616703567281cb8ull, \
  0x56344b525f1ff495ull, \
  0x565230ca0904d3f6ull, \
  0x5670209ffc1f2e82ull, \
  0x568e1ad7d0f6487eull, \
  0x56ac1f752150a563ull, \
  0x56ca2e7b88347698ull, \
  0x56e847eea1e80a49ull, \
  0x57066bd20bf23a72ull, \
  0x57249a29651adc07ull, \
  0x5742d2f84d6b2e47ull, \
  0x57611642662e4a33ull, \
  0x577f640b51f1922bull, \
  0x579dbc56b48521baull, \
  0x57bc1f2832fc3d7bull, \
  0x57da8c8373adc331ull, \
  0x57f9046c1e3499fcull, \
  0x581786e5db7022c2ull, \
  0x583613f45584a8aeull, \
  0x5854ab9b37dbd1e5ull, \
  0x58734dde2f251059ull, \
  0x5891fac0e95612c8ull, \
  0x58b0b24715ab35deull, \
  0x58cf747464a7f584ull, \
  0x58ee414c88175e50ull, \
  0x590d18d3330c7f1eull, \
  0x592bfb0c19e2dad6ull, \
  0x594ae7faf23eda52ull, \
  0x5969dfa3730e3e6full, \
  0x5988e20954889245ull, \
  0x59a7ef30502f9d87ull, \
  0x59c7071c20cfd70cull, \
  0x59e629d08280d77aull, \
  0x5a05575132a5cc20ull, \
  0x5a248fa1efede9f7ull, \
  0x5a43d2c67a54e0c0ull, \
  0x5a6320c293234e5eull, \
  0x5a827999fcef3242ull, \
  0x5aa1dd507b9c6112ull, \
  0x5ac14be9d45cf869ull, \
  0x5ae0c569cdb1d2caull, \
  0x5b0049d42f6afbb6ull, \
  0x5b1fd92cc2a823eaull, \
  0x5b3f737751d915c8ull, \
  0x5b5f18b7a8be29e6ull, \
  0x5b7ec8f19468bbc9ull, \
  0x5b9e8428e33b9ec0ull, \
  0x5bbe4a6164eb92f4ull, \
  0x5bde1b9eea7fba97ull, \
  0x5bfdf7e546520f3eull, \
  0x5c1ddf384c0fd764ull, \
  0x5c3dd19bd0ba1c1aull, \
  0x5c5dcf13aaa61ed5ull, \
  0x5c7dd7a3b17dcf75ull, \
  0x5c9deb4fbe404261ull, \
  0x5cbe0a1bab4226dfull, \
  0x5cde340b542e3d8bull, \
  0x5cfe69229605cef5ull, \
  0x5d1ea9654f212270ull, \
  0x5d3ef4d75f2ff504ull, \
  0x5d5f4b7ca739f08dull, \
  0x5d7fad59099f22feull, \
  0x5da01a706a1875d6ull, \
  0x5dc092c6adb825b8ull, \
  0x5de1165fbaea3a2aull, \
  0x5e01a53f7974fd86ull, \
  0x5e223f69d2797511ull, \
  0x5e42e4e2b073d935ull, \
  0x5e6395adff3c0deeull, \
  0x5e8451cfac061b5full, \
  0x5ea5194ba562a68cull, \
  0x5ec5ec25db3f6a41ull, \
  0x5ee6ca623ee7b025ull, \
  0x5f07b404c304c9f1ull, \
  0x5f28a9115b9e8adaull, \
  0x5f49a98bfe1bc11cull, \
  0x5f6ab578a142afb3ull, \
  0x5f8bccdb3d398841ull, \
  0x5facefb7cb86e51bull, \
  0x5fce1e124712437cull, \
  0x5fef57eeac247df0ull, \
  0x60109d50f86846d8ull, \
  0x6031ee3d2aeaa329ull, \
  0x60534ab7441b6546ull, \
  0x6074b2c345cda814ull, \
  0x6096266533384a2bull, \
  0x60b7a5a110f6693cull, \
  0x60d9307ae507dd9aull, \
  0x60fac6f6b6d1b5f5ull, \
  0x611c69188f1eb339ull, \
  0x613e16e4781fc4a0ull, \
  0x615fd05e7d6c83e4ull, \
  0x6181958aac03b1a8ull, \
  0x61a3666d124bb204ull, \
  0x61c54309c013093dull, \
  0x61e72b64c690d8afull, \
  0x62091f8238655bd8ull, \
  0x622b1f66299a6599ull, \
  0x624d2b14afa3dd98ull, \
  0x626f4291e1603dd5ull, \
  0x629165e1d7191069ull, \
  0x62b39508aa836d6full, \
  0x62d5d00a76c07917ull, \
  0x62f816eb585de1edull, \
  0x631a69af6d565f3full, \
  0x633cc85ad5122fbdull, \
  0x635f32f1b0679836ull, \
  0x6381a978219b628full, \
  0x63a42bf24c615cddull, \
  0x63c6ba6455dcd8aeull, \
  0x63e954d264a12a7full, \
  0x640bfb40a0b22959ull, \
  0x642eadb33384aea6ull, \
  0x64516c2e47ff1623ull, \
  0x647436b60a79be0aull, \
  0x64970d4ea8bf8766ull, \
  0x64b9effc520e568dull, \
  0x64dcdec3371793d1ull, \
  0x64ffd9a78a00ac55ull, \
  0x6522e0ad7e639312ull, \
  0x6545f3d9494f420aull, \
  0x6569132f21483ba7ull, \
  0x658c3eb33e490c43ull, \
  0x65af7669d9c2cbe4ull, \
  0x65d2ba572e9da020ull, \
  0x65f60a7f79393e2eull, \
  0x661966e6f76d6d28ull, \
  0x663ccf91e88a8873ull, \
  0x666044848d5a025eull, \
  0x6683c5c3281ee6e9ull, \
  0x66a75351fc965eb3ull, \
  0x66caed354ff83222ull, \
  0x66ee937168f74cb3ull, \
  0x6712460a8fc24072ull, \
  0x673605050e03c9a7ull, \
  0x6759d0652ee352afull, \
  0x677da82f3f057800ull, \
  0x67a18c678c8c8c61ull, \
  0x67c57d1267191d43ull, \
  0x67e97a341fca775bull, \
  0x680d83d1093f2b56ull, \
  0x683199ed779592caull, \
  0x6855bc8dc06c5550ull, \
  0x6879ebb63ae2edc6ull, \
  0x689e276b3f9a2fccull, \
  0x68c26fb128b4cd63ull, \
  0x68e6c48c51d7dcc2ull, \
  0x690b2601182b5e56ull, \
  0x692f9413da5ac2f2ull, \
  0x69540ec8f895722dull, \
  0x69789624d48f50efull, \
  0x699d2a2bd181482aull, \
  0x69c1cae25429cbc7ull, \
  0x69e6784cc2cd61bdull, \
  0x6a0b326f85372957ull, \
  0x6a2ff94f04b962b0ull, \
  0x6a54ccefac2df653ull, \
  0x6a79ad55e7f6fd10ull, \
  0x6a9e9a8625ff4803ull, \
  0x6ac39484d5bae8c5ull, \
  0x6ae89b566827b9cdull, \
  0x6b0daeff4fcde703ull, \
  0x6b32cf8400c07681ull, \
  0x6b57fce8f09dd17full, \
  0x6b7d373296904d79ull, \
  0x6ba27e656b4eb57aull, \
  0x6bc7d285e91cd39cull, \
  0x6bed33988bcbfab5ull, \
  0x6c12a1a1d0bb9038ull, \
  0x6c381ca636d99642ull, \
  0x6c5da4aa3ea335d6ull, \
  0x6c8339b26a25494eull, \
  0x6ca8dbc33cfce6f5ull, \
  0x6cce8ae13c57ebdbull, \
  0x6cf44710eef586ccull, \
  0x6d1a1056dd26c382ull, \
  0x6d3fe6b790cf1606ull, \
  0x6d65ca379564e639ull, \
  0x6d8bbadb77f21b98ull, \
  0x6db1b8a7c714a92bull, \
  0x6dd7c3a112ff19a2ull, \
  0x6dfddbcbed791babull, \
  0x6e24012ce9e00e6full, \
  0x6e4a33c89d278e49ull, \
  0x6e7073a39dda01a3ull, \
  0x6e96c0c284192610ull, \
  0x6ebd1b29e99e9d8dull, \
  0x6ee382de69bc7bf8ull, \
  0x6f09f7e4a15dd4b8ull, \
  0x6f307a412f074892ull, \
  0x6f5709f8b2d793b7ull, \
  0x6f7da70fce881bf9ull, \
  0x6fa4518b256d7f3cull, \
  0x6fcb096f5c782210ull, \
  0x6ff1cec11a34be80ull, \
  0x7018a18506ccf314ull, \
  0x703f81bfcc07d1ffull, \
  0x70666f76154a7089ull, \
  0x708d6aac8f98769cull, \
  0x70b47367e994ae92ull, \
  0x70db89acd381952aull, \
  0x7102ad7fff41e9b4ull, \
  0x7129dee620593e6full, \
  0x71511de3ebec8913ull, \
  0x71786a7e18c2b399ull, \
  0x719fc4b95f452d29ull, \
  0x71c72c9a79807b40ull, \
  0x71eea2262324cb0cull, \
  0x72162561198682f1ull, \
  0x723db6501b9ed447ull, \
  0x726554f7ea0c4d4bull, \
  0x728d015d47136b40ull, \
  0x72b4bb84f69f2cc4ull, \
  0x72dc8373be41a454ull, \
  0x7304592e65348b0bull, \
  0x732c3cb9b459d38bull, \
  0x73542e1a763c3d21ull, \
  0x737c2d55770fe711ull, \
  0x73a43a6f84b2e425ull, \
  0x73cc556d6eadce5full, \
  0x73f47e5406345aeaull, \
  0x741cb5281e25ee34ull, \
  0x7444f9ee8b0e304aull, \
  0x746d4cac2325a155ull, \
  0x7495ad65be522e5cull, \
  0x74be1c203627c62bull, \
  0x74e698e065e8ee7aull, \
  0x750f23ab2a87593eull, \
  0x7537bc8562a47a32ull, \
  0x75606373ee921c97ull, \
  0x7589187bb052f922ull, \
  0x75b1dba18b9b4c20ull, \
  0x75daacea65d16bcfull, \
  0x76038c5b260e5eeeull, \
  0x762c79f8b51e7379ull, \
  0x765575c7fd81d5a0ull, \
  0x767e7fcdeb6d26f5ull, \
  0x76a7980f6cca15c2ull, \
  0x76d0be917137f4a3ull, \
  0x76f9f358ea0c5249ull, \
  0x7723366aca539175ull, \
  0x774c87cc06d1812eull, \
  0x7775e7819601f51full, \
  0x779f559070195e36ull, \
  0x77c8d1fd8f056372ull, \
  0x77f25ccdee6d7ae6ull, \
  0x781bf6068bb382f3ull, \
  0x78459dac65f45bb5ull, \
  0x786f53c47e0880aaull, \
  0x78991853d684a285ull, \
  0x78c2eb5f73ba4140ull, \
  0x78ecccec5bb84661ull, \
  0x7916bcff964b9f6dull, \
  0x7940bb9e2cffd89dull, \
  0x796ac8cd2b1fb7beull, \
  0x7994e4919db5d74eull, \
  0x79bf0ef0938d41c8ull, \
  0x79e947ef1d320d2dull, \
  0x7a138f924cf1f6bfull, \
  0x7a3de5df36dcfeefull, \
  0x7a684adaf0c6058bull, \
  0x7a92be8a92436616ull, \
  0x7abd40f334af945eull, \
  0x7ae7d219f329b948ull, \
  0x7b127203ea964fceull, \
  0x7b3d20b6399fc237ull, \
  0x7b67de3600b70786ull, \
  0x7b92aa886214411cull, \
  0x7bbd85b281b75897ull, \
  0x7be86fb985689ddcull, \
  0x7c1368a294b9656aull, \
  0x7c3e7072d904a6ceull, \
  0x7c69872f7d6f9b63ull, \
  0x7c94acddaeea5d3aull, \
  0x7cbfe1829c308640ull, \
  0x7ceb252375c9cf9bull, \
  0x7d1677c56e0ab138ull, \
  0x7d41d96db915019dull, \
  0x7d6d4a218cd895e5ull, \
  0x7d98c9e62113e1faull, \
  0x7dc458c0af549908ull, \
  0x7deff6b672f84e24ull, \
  0x7e1ba3cca92d152cull, \
  0x7e47600890f223deull, \
  0x7e732b6f6b18732aull, \
  0x7e9f06067a4360baull, \
  0x7ecaefd302e950afull, \
  0x7ef6e8da4b544f9aull, \
  0x7f22f1219ba2b4aeull, \
  0x7f4f08ae3dc7c426ull, \
  0x7f7b2f857d8c51e5ull, \
  0x7fa765aca88f6453ull, \
  0x7fd3ab290e46d769ull, \
}

// per 9-bit significand interval: {c, (-log(c/2048) - 1100 ln2) 2^72 in three words, lowest first}
#define FM_LOG_TABLE_INIT { \
  {2048u, 0x8131d882u, 0xc1032678u, 0xfffd0589u}, \
  {2045u, 0xc5932a1fu, 0x21152af9u, 0xfffd058au}, \
  {2041u, 0xca32846bu, 0xa1655fc8u, 0xfffd058au}, \
  {2037u, 0x974d40b7u, 0x21f60533u, 0xfffd058bu}, \
  {2033u, 0x2f0180a7u, 0xa2c75c14u, 0xfffd058bu}, \
  {2029u, 0xaaeab54au, 0x23d9a5a6u, 0xfffd058cu}, \
  {2025u, 0x0258ffdfu, 0xa52d238au, 0xfffd058cu}, \
  {2021u, 0xd27e3cfcu, 0x26c217c0u, 0xfffd058du}, \
  {2017u, 0x2896b0beu, 0xa898c4b2u, 0xfffd058du}, \
  {2013u, 0x4e135fcfu, 0x2ab16d2au, 0xfffd058eu}, \
  {2009u, 0x96cc36a5u, 0xad0c545bu, 0xfffd058eu}, \
  {2005u, 0x31403644u, 0x2fa9bddfu, 0xfffd058fu}, \
  {2002u, 0x82e67f13u, 0x91cb9b6cu, 0xfffd058fu}, \
  {1998u, 0x124f377bu, 0x14de0ce1u, 0xfffd0590u}, \
  {1994u, 0x476b5cf0u, 0x9833bca6u, 0xfffd0590u}, \
  {1990u, 0x67325d31u, 0x1bccefdeu, 0xfffd0591u}, \
  {1986u, 0x8b474515u, 0x9fa9ec16u, 0xfffd0591u}, \
  {1983u, 0x4064202eu, 0x02bc4f3cu, 0xfffd0592u}, \
  {1979u, 0x5a5487cfu, 0x871093d4u, 0xfffd0592u}, \
  {1975u, 0x683f2217u, 0x0ba962deu, 0xfffd0593u}, \
  {1972u, 0x196755e1u, 0x6f4923c9u, 0xfffd0593u}, \
  {1968u, 0x73269ec7u, 0xf45a908fu, 0xfffd0593u}, \
  {1964u, 0x68a94aa2u, 0x79b14c7au, 0xfffd0594u}, \
  {1960u, 0xdeddf904u, 0xff4d9fe2u, 0xfffd0594u}, \
  {1957u, 0x0ae4656du, 0x63b0b5a1u, 0xfffd0595u}, \
  {1953u, 0xf965e30au, 0xe9c78190u, 0xfffd0595u}, \
  {1950u, 0x3abbe732u, 0x4e86c5f7u, 0xfffd0596u}, \
  {1946u, 0x31ea2bc1u, 0xd518ebc2u, 0xfffd0596u}, \
  {1942u, 0xde884d58u, 0x5bf1f424u, 0xfffd0597u}, \
  {1939u, 0x0339592eu, 0xc1436c22u, 0xfffd0597u}, \
  {1935u, 0xb4bfd162u, 0x48993565u, 0xfffd0598u}, \
  {1932u, 0x7859024fu, 0xae4894acu, 0xfffd0598u}, \
  {1928u, 0xdd6fb0b8u, 0x361c067bu, 0xfffd0599u}, \
  {1924u, 0x4ab21eceu, 0xbe37af4eu, 0xfffd0599u}, \
  {1921u, 0xa5443c9bu, 0x247c004bu, 0xfffd059au}, \
  {1917u, 0x27326a7bu, 0xad16c2d6u, 0xfffd059au}, \
  {1914u, 0xbdfa7361u, 0x13bac033u, 0xfffd059bu}, \
  {1910u, 0x9a3cfd5bu, 0x9cd58ab5u, 0xfffd059bu}, \
  {1907u, 0x0b8df4d8u, 0x03d9e81eu, 0xfffd059cu}, \
  {1904u, 0x98d6642au, 0x6b07cabfu, 0xfffd059cu}, \
  {1900u, 0xc07d42ccu, 0xf4db1e90u, 0xfffd059cu}, \
  {1897u, 0xc4808bf7u, 0x5c6a655au, 0xfffd059du}, \
  {1893u, 0xcae4aeabu, 0xe6c00ebfu, 0xfffd059du}, \
  {1890u, 0x914a33a2u, 0x4eb1723bu, 0xfffd059eu}, \
  {1886u, 0x943bf618u, 0xd98a689eu, 0xfffd059eu}, \
  {1883u, 0xd833d635u, 0x41dea363u, 0xfffd059fu}, \
  {1880u, 0x12fd5563u, 0xaa5d7410u, 0xfffd059fu}, \
  {1876u, 0xdbab71ceu, 0x35f3afaeu, 0xfffd05a0u}, \
  {1873u, 0xfea75bc3u, 0x9ed665d4u, 0xfffd05a0u}, \
  {1870u, 0xf00b0713u, 0x07e4269au, 0xfffd05a1u}, \
  {1866u, 0x14fa64c0u, 0x9439ae3bu, 0xfffd05a1u}, \
  {1863u, 0x2ac53cedu, 0xfdac6705u, 0xfffd05a1u}, \
  {1860u, 0x5d5a9931u, 0x674aa10au, 0xfffd05a2u}, \
  {1856u, 0xcaba869fu, 0xf46183d1u, 0xfffd05a2u}, \
  {1853u, 0x3aa0646eu, 0x5e65ccd7u, 0xfffd05a3u}, \
  {1850u, 0xfdde3ba8u, 0xc8960f9fu, 0xfffd05a3u}, \
  {1847u, 0xa820fda0u, 0x32f270b6u, 0xfffd05a4u}, \
  {1843u, 0x07ddbe42u, 0xc107d293u, 0xfffd05a4u}, \
  {1840u, 0xdc4db877u, 0x2bcbb425u, 0xfffd05a5u}, \
  {1837u, 0xaa4d2d9fu, 0x96bc2f1fu, 0xfffd05a5u}, \
  {1834u, 0xdde2ea9fu, 0x01d968d2u, 0xfffd05a6u}, \
  {1830u, 0x94d9fbb1u, 0x90f0e666u, 0xfffd05a6u}, \
  {1827u, 0xa0cc591cu, 0xfc7719f6u, 0xfffd05a6u}, \
  {1824u, 0xc7d4288au, 0x682a89fcu, 0xfffd05a7u}, \
  {1821u, 0x0a094dfeu, 0xd40b5c99u, 0xfffd05a7u}, \
  {1818u, 0xae7012e6u, 0x4019b81bu, 0xfffd05a8u}, \
  {1815u, 0x949e2494u, 0xac55c305u, 0xfffd05a8u}, \
  {1812u, 0x870c73a9u, 0x18bfa408u, 0xfffd05a9u}, \
  {1808u, 0x56976d5au, 0xa9946054u, 0xfffd05a9u}, \
  {1805u, 0xcd190a30u, 0x1669cc76u, 0xfffd05aau}, \
  {1802u, 0x17621eaau, 0x836d9113u, 0xfffd05aau}, \
  {1799u, 0xc1cb9298u, 0xf09fd5b2u, 0xfffd05aau}, \
  {1796u, 0x064b23edu, 0x5e00c212u, 0xfffd05abu}, \
  {1793u, 0x2334ebecu, 0xcb907e20u, 0xfffd05abu}, \
  {1790u, 0xb2b6d995u, 0x394f31ffu, 0xfffd05acu}, \
  {1787u, 0x0310004fu, 0xa73d0607u, 0xfffd05acu}, \
  {1784u, 0x6f859fa4u, 0x155a22c0u, 0xfffd05adu}, \
  {1781u, 0xba17ce77u, 0x83a6b0eau, 0xfffd05adu}, \
  {1778u, 0x65f7ba02u, 0xf222d979u, 0xfffd05adu}, \
  {1775u, 0x12c16ea8u, 0x60cec595u, 0xfffd05aeu}, \
  {1772u, 0xd87b26b7u, 0xcfaa9e9bu, 0xfffd05aeu}, \
  {1769u, 0xa45c212bu, 0x3eb68e21u, 0xfffd05afu}, \
  {1766u, 0x965d08a3u, 0xadf2bdf0u, 0xfffd05afu}, \
  {1763u, 0x5f93f8eeu, 0x1d5f5809u, 0xfffd05b0u}, \
  {1760u, 0xa15e37d2u, 0x8cfc86a3u, 0xfffd05b0u}, \
  {1757u, 0x4d59bc1bu, 0xfcca742eu, 0xfffd05b0u}, \
  {1754u, 0x0630a463u, 0x6cc94b50u, 0xfffd05b1u}, \
  {1751u, 0x8138c597u, 0xdcf936e7u, 0xfffd05b1u}, \
  {1748u, 0xe8e97fdbu, 0x4d5a620bu, 0xfffd05b2u}, \
  {1745u, 0x402a0f26u, 0xbdecf80du, 0xfffd05b2u}, \
  {1742u, 0xc67a93bfu, 0x2eb12474u, 0xfffd05b3u}, \
  {1739u, 0x5cfa15a3u, 0x9fa71305u, 0xfffd05b3u}, \
  {1737u, 0x719cea6eu, 0xeb116c88u, 0xfffd05b3u}, \
  {1734u, 0x8cd557f4u, 0x5c5aab3au, 0xfffd05b4u}, \
  {1731u, 0xdb1444e8u, 0xcdd621e4u, 0xfffd05b4u}, \
  {1728u, 0xfc95cf87u, 0x3f83fd20u, 0xfffd05b5u}, \
  {1725u, 0x1654411bu, 0xb16469c4u, 0xfffd05b5u}, \
  {1722u, 0x3c1e5b2eu, 0x237794dfu, 0xfffd05b6u}, \
  {1719u, 0xdb9a6bbcu, 0x95bdabbfu, 0xfffd05b6u}, \
  {1717u, 0xf002cc12u, 0xe208c63du, 0xfffd05b6u}, \
  {1714u, 0x00c00896u, 0x54a420b9u, 0xfffd05b7u}, \
  {1711u, 0x4966e447u, 0xc772e0f2u, 0xfffd05b7u}, \
  {1708u, 0x23cb2f75u, 0x3a753518u, 0xfffd05b8u}, \
  {1706u, 0x363e199eu, 0x873e2b9fu, 0xfffd05b8u}, \
  {1703u, 0xc8b20c8fu, 0xfa96dd98u, 0xfffd05b8u}, \
  {1700u, 0x36d1a2f6u, 0x6e239fd7u, 0xfffd05b9u}, \
  {1697u, 0xa141cc87u, 0xe1e4a16fu, 0xfffd05b9u}, \
  {1694u, 0x238f5857u, 0x55da11b7u, 0xfffd05bau}, \
  {1692u, 0x545ac3c5u, 0xa345951au, 0xfffd05bau}, \
  {1689u, 0xc7518696u, 0x1792d263u, 0xfffd05bbu}, \
  {1686u, 0xdcaf352du, 0x8c14fdd0u, 0xfffd05bbu}, \
  {1684u, 0xfae45b24u, 0xd9de9a71u, 0xfffd05bbu}, \
  {1681u, 0x58014ef6u, 0x4eb968d1u, 0xfffd05bcu}, \
  {1678u, 0xd61cb620u, 0xc3c9a69bu, 0xfffd05bcu}, \
  {1676u, 0xd5a2d2c1u, 0x11f2424fu, 0xfffd05bdu}, \
  {1673u, 0x9f90663eu, 0x875bfc0eu, 0xfffd05bdu}, \
  {1670u, 0xf113c981u, 0xfcfba85bu, 0xfffd05bdu}, \
  {1668u, 0xd73c504au, 0x4b842c45u, 0xfffd05beu}, \
  {1665u, 0x3f3baa0au, 0xc17e30aau, 0xfffd05beu}, \
  {1662u, 0xa88b7db7u, 0x37aeaca5u, 0xfffd05bfu}, \
  {1660u, 0xd8daae30u, 0x86980546u, 0xfffd05bfu}, \
  {1657u, 0x60d1dea7u, 0xfd23b8acu, 0xfffd05bfu}, \
  {1654u, 0xdae6e705u, 0x73e66a9fu, 0xfffd05c0u}, \
  {1652u, 0xc8d5f290u, 0xc33187e8u, 0xfffd05c0u}, \
  {1649u, 0x7e321e6cu, 0x3a5053d9u, 0xfffd05c1u}, \
  {1647u, 0xd6376a13u, 0x89d90770u, 0xfffd05c1u}, \
  {1644u, 0x749ad10fu, 0x01547ca8u, 0xfffd05c2u}, \
  {1641u, 0xc87daddfu, 0x7907cff6u, 0xfffd05c2u}, \
  {1639u, 0xb6b91882u, 0xc8f3d59bu, 0xfffd05c2u}, \
  {1636u, 0xf9d6826au, 0x4104ba2eu, 0xfffd05c3u}, \
  {1634u, 0xb44182b1u, 0x912f5176u, 0xfffd05c3u}, \
  {1631u, 0x2e19b088u, 0x099e5a09u, 0xfffd05c4u}, \
  {1629u, 0x3f70dca3u, 0x5a07e538u, 0xfffd05c4u}, \
  {1626u, 0x69d2b07fu, 0xd2d5a5deu, 0xfffd05c4u}, \
  {1624u, 0x93b24306u, 0x237e8821u, 0xfffd05c5u}, \
  {1621u, 0x5f32fdd5u, 0x9cab964eu, 0xfffd05c5u}, \
  {1619u, 0x78006e3cu, 0xed9433bdu, 0xfffd05c5u}, \
  {1616u, 0xa155fcd0u, 0x67212646u, 0xfffd05c6u}, \
  {1614u, 0x7d85fabdu, 0xb849e3e7u, 0xfffd05c6u}, \
  {1611u, 0xf41447f6u, 0x32375309u, 0xfffd05c7u}, \
  {1609u, 0x5b034af1u, 0x83a096d3u, 0xfffd05c7u}, \
  {1606u, 0xb8eec2efu, 0xfdef1c37u, 0xfffd05c7u}, \
  {1604u, 0x65838e90u, 0x4f994d14u, 0xfffd05c8u}, \
  {1601u, 0x799cca55u, 0xca4983d3u, 0xfffd05c8u}, \
  {1599u, 0x26ed7d1fu, 0x1c3509a5u, 0xfffd05c9u}, \
  {1597u, 0x97738181u, 0x6e3acec0u, 0xfffd05c9u}, \
  {1594u, 0x12ff65eau, 0xe974d1efu, 0xfffd05c9u}, \
  {1592u, 0x9b75b57cu, 0x3bbc7f13u, 0xfffd05cau}, \
  {1589u, 0x5b496091u, 0xb759add2u, 0xfffd05cau}, \
  {1587u, 0x3ec07e29u, 0x09e3ad3fu, 0xfffd05cbu}, \
  {1584u, 0xe2bba633u, 0x85e4a7adu, 0xfffd05cbu}, \
  {1582u, 0x1f8f29c1u, 0xd8b164a4u, 0xfffd05cbu}, \
  {1580u, 0x9c827a63u, 0x2b98f213u, 0xfffd05ccu}, \
  {1577u, 0xe5767594u, 0xa826b32cu, 0xfffd05ccu}, \
  {1575u, 0xbe36a631u, 0xfb519604u, 0xfffd05ccu}, \
  {1573u, 0x0e5e7a47u, 0x4e97867du, 0xfffd05cdu}, \
  {1570u, 0xb1a1f992u, 0xcbb34f4fu, 0xfffd05cdu}, \
  {1568u, 0x13215150u, 0x1f3d2f18u, 0xfffd05ceu}, \
  {1566u, 0x461e7da4u, 0x72e25a7au, 0xfffd05ceu}, \
  {1563u, 0x34820812u, 0xf08d7064u, 0xfffd05ceu}, \
  {1561u, 0x387d5c0bu, 0x44772710u, 0xfffd05cfu}, \
  {1559u, 0x51f254cfu, 0x987c6825u, 0xfffd05cfu}, \
  {1556u, 0x8d1b541fu, 0x16b814e7u, 0xfffd05d0u}, \
  {1554u, 0xce2cddcdu, 0x6b027f5bu, 0xfffd05d0u}, \
  {1552u, 0x2f854f2au, 0xbf68b3e2u, 0xfffd05d0u}, \
  {1549u, 0x11e61786u, 0x3e3645b5u, 0xfffd05d1u}, \
  {1547u, 0x4c9d4282u, 0x92e243d5u, 0xfffd05d1u}, \
  {1545u, 0x6c927ef9u, 0xe7aa4c8eu, 0xfffd05d1u}, \
  {1543u, 0x61a23505u, 0x3c8e7279u, 0xfffd05d2u}, \
  {1540u, 0x6a55f439u, 0xbc198af3u, 0xfffd05d2u}, \
  {1538u, 0xdc4f5343u, 0x11444bb1u, 0xfffd05d3u}, \
  {1536u, 0xef7bb971u, 0x668b6b4bu, 0xfffd05d3u}, \
  {1534u, 0xb3a51481u, 0xbbeefcaeu, 0xfffd05d3u}, \
  {1531u, 0x69404ef9u, 0x3c39d5b0u, 0xfffd05d4u}, \
  {1529u, 0xbd6226f6u, 0x91e4d6d2u, 0xfffd05d4u}, \
  {1527u, 0x7630fa52u, 0xe7ac8c91u, 0xfffd05d4u}, \
  {1525u, 0xc1c66e40u, 0x3d910a2fu, 0xfffd05d5u}, \
  {1522u, 0x2883062du, 0xbe9de7b3u, 0xfffd05d5u}, \
  {1520u, 0xf4c09b18u, 0x14caadc5u, 0xfffd05d6u}, \
  {1518u, 0x03d0fd84u, 0x6b147fbdu, 0xfffd05d6u}, \
  {1516u, 0xafb5652cu, 0xc17b7133u, 0xfffd05d6u}, \
  {1514u, 0x335d0abdu, 0x17ff95d9u, 0xfffd05d7u}, \
  {1511u, 0xd2bcf7abu, 0x99fcb809u, 0xfffd05d7u}, \
  {1509u, 0x7b05ab05u, 0xf0ca3346u, 0xfffd05d7u}, \
  {1507u, 0x5ac0a7bbu, 0x47b52735u, 0xfffd05d8u}, \
  {1505u, 0x709d77b4u, 0x9ebda7e0u, 0xfffd05d8u}, \
  {1503u, 0x327137e2u, 0xf5e3c966u, 0xfffd05d8u}, \
  {1501u, 0xa91e41c7u, 0x4d279ff9u, 0xfffd05d9u}, \
  {1498u, 0x1fa0cdf6u, 0xd04541b3u, 0xfffd05d9u}, \
  {1496u, 0x244e5f5fu, 0x27d3b5d0u, 0xfffd05dau}, \
  {1494u, 0x1a381c91u, 0x7f802651u, 0xfffd05dau}, \
  {1492u, 0xfe54ad6fu, 0xd74aa7c6u, 0xfffd05dau}, \
  {1490u, 0xfd7fb465u, 0x2f334ed7u, 0xfffd05dbu}, \
  {1488u, 0x919df17du, 0x873a303fu, 0xfffd05dbu}, \
  {1486u, 0x9ef390c8u, 0xdf5f60ceu, 0xfffd05dbu}, \
  {1484u, 0x91ad0bcfu, 0x37a2f56bu, 0xfffd05dcu}, \
  {1482u, 0x7b9b06e1u, 0x90050312u, 0xfffd05dcu}, \
  {1479u, 0x87b136d0u, 0x14d1689cu, 0xfffd05ddu}, \
  {1477u, 0x4741ea53u, 0x6d80013au, 0xfffd05ddu}, \
  {1475u, 0x66d1315cu, 0xc64d5d00u, 0xfffd05ddu}, \
  {1473u, 0xd6f32b92u, 0x1f39914du, 0xfffd05deu}, \
  {1471u, 0xd50b62aau, 0x7844b397u, 0xfffd05deu}, \
  {1469u, 0x0a5e4bb2u, 0xd16ed96au, 0xfffd05deu}, \
  {1467u, 0xab58f62fu, 0x2ab81866u, 0xfffd05dfu}, \
  {1465u, 0x970f5abcu, 0x84208646u, 0xfffd05dfu}, \
  {1463u, 0x76f1bb9du, 0xdda838d9u, 0xfffd05dfu}, \
  {1461u, 0xdeb98b23u, 0x374f4605u, 0xfffd05e0u}, \
  {1459u, 0x6c8e4c98u, 0x9115c3c9u, 0xfffd05e0u}, \
  {1457u, 0xe962e5bbu, 0xeafbc838u, 0xfffd05e0u}, \
  {1455u, 0x698bd7ceu, 0x45016980u, 0xfffd05e1u}, \
  {1453u, 0x6d8ed883u, 0x9f26bde3u, 0xfffd05e1u}, \
  {1451u, 0x032c4417u, 0xf96bdbbdu, 0xfffd05e1u}, \
  {1449u, 0xe6a2e33fu, 0x53d0d97fu, 0xfffd05e2u}, \
  {1447u, 0xa42e8096u, 0xae55cdb6u, 0xfffd05e2u}, \
  {1445u, 0xb9c1ca83u, 0x08facf03u, 0xfffd05e3u}, \
  {1443u, 0xb8fbffbdu, 0x63bff421u, 0xfffd05e3u}, \
  {1441u, 0x695ae5d4u, 0xbea553e3u, 0xfffd05e3u}, \
  {1439u, 0xeaa98a4du, 0x19ab0533u, 0xfffd05e4u}, \
  {1437u, 0xd7ac5049u, 0x74d11f16u, 0xfffd05e4u}, \
  {1435u, 0x690acdbcu, 0xd017b8a8u, 0xfffd05e4u}, \
  {1433u, 0x9877fcb8u, 0x2b7ee91du, 0xfffd05e5u}, \
  {1431u, 0x4419466du, 0x8706c7c4u, 0xfffd05e5u}, \
  {1429u, 0x522ceef9u, 0xe2af6c03u, 0xfffd05e5u}, \
  {1427u, 0xd4f06a46u, 0x3e78ed5au, 0xfffd05e6u}, \
  {1425u, 0x2ec723bcu, 0x9a636364u, 0xfffd05e6u}, \
  {1423u, 0x36a243bfu, 0xf66ee5d2u, 0xfffd05e6u}, \
  {1421u, 0x5ca9ff6du, 0x529b8c71u, 0xfffd05e7u}, \
  {1419u, 0xcf29005au, 0xaee96f27u, 0xfffd05e7u}, \
  {1417u, 0x9fba7384u, 0x0b58a5f5u, 0xfffd05e8u}, \
  {1416u, 0x6e281719u, 0x399cc86cu, 0xfffd05e8u}, \
  {1414u, 0x6a4db937u, 0x963e2a96u, 0xfffd05e8u}, \
  {1412u, 0x2968544au, 0xf3011d4au, 0xfffd05e8u}, \
  {1410u, 0x81473653u, 0x4fe5b8e3u, 0xfffd05e9u}, \
  {1408u, 0xd5a1901eu, 0xacec15d8u, 0xfffd05e9u}, \
  {1406u, 0x3ebd5b58u, 0x0a144cbbu, 0xfffd05eau}, \
  {1404u, 0xb05caddfu, 0x675e7636u, 0xfffd05eau}, \
  {1402u, 0x20f2145fu, 0xc4caab12u, 0xfffd05eau}, \
  {1400u, 0xb11c901bu, 0x2259042fu, 0xfffd05ebu}, \
  {1399u, 0x668b5ba0u, 0x512d0625u, 0xfffd05ebu}, \
  {1397u, 0xf16fb537u, 0xaeeec489u, 0xfffd05ebu}, \
  {1395u, 0xcba47a21u, 0x0cd2e5ddu, 0xfffd05ecu}, \
  {1393u, 0x646d71e4u, 0x6ad98363u, 0xfffd05ecu}, \
  {1391u, 0x0a6fefe7u, 0xc902b679u, 0xfffd05ecu}, \
  {1389u, 0x14c3f8d3u, 0x274e9899u, 0xfffd05edu}, \
  {1388u, 0xef3fbaf8u, 0x5681934au, 0xfffd05edu}, \
  {1386u, 0xabb3629au, 0xb501abfdu, 0xfffd05edu}, \
  {1384u, 0x5b582b36u, 0x13a4b3e8u, 0xfffd05eeu}, \
  {1382u, 0xba8a0689u, 0x726ac4e8u, 0xfffd05eeu}, \
  {1380u, 0x4a979966u, 0xd153f8f9u, 0xfffd05eeu}, \
  {1378u, 0x7c7c2dc0u, 0x30606a31u, 0xfffd05efu}, \
  {1377u, 0xb98c7fb8u, 0x5ff3e1ebu, 0xfffd05efu}, \
  {1375u, 0x08513304u, 0xbf35600bu, 0xfffd05efu}, \
  {1373u, 0x47275b05u, 0x1e9a5d0cu, 0xfffd05f0u}, \
  {1371u, 0x82dfed27u, 0x7e22f36du, 0xfffd05f0u}, \
  {1369u, 0x7c1e5434u, 0xddcf3dcau, 0xfffd05f0u}, \
  {1368u, 0x361e0979u, 0x0db2ced0u, 0xfffd05f1u}, \
  {1366u, 0x3bb69255u, 0x6d94d94cu, 0xfffd05f1u}, \
  {1364u, 0x77c3c829u, 0xcd9adaccu, 0xfffd05f1u}, \
  {1362u, 0x009b8519u, 0x2dc4ee56u, 0xfffd05f2u}, \
  {1361u, 0x2e247151u, 0x5de78758u, 0xfffd05f2u}, \
  {1359u, 0xf5565499u, 0xbe47e8dbu, 0xfffd05f2u}, \
  {1357u, 0x8f3d6e6au, 0x1ecca07bu, 0xfffd05f3u}, \
  {1355u, 0x96bf230eu, 0x7f75c9a7u, 0xfffd05f3u}, \
  {1354u, 0xf5b291a2u, 0xafd8116du, 0xfffd05f3u}, \
  {1352u, 0xe8bf9531u, 0x10b818a3u, 0xfffd05f4u}, \
  {1350u, 0x6388cab9u, 0x71bcd688u, 0xfffd05f4u}, \
  {1348u, 0xc2ede70eu, 0xd2e666f9u, 0xfffd05f4u}, \
  {1347u, 0x749504dcu, 0x038906e5u, 0xfffd05f5u}, \
  {1345u, 0xaa726d4cu, 0x64ea07b0u, 0xfffd05f5u}, \
  {1343u, 0x1f72a1f0u, 0xc6702140u, 0xfffd05f5u}, \
  {1341u, 0x3edd22c6u, 0x281b6fe2u, 0xfffd05f6u}, \
  {1340u, 0xadea08e5u, 0x58ff13fbu, 0xfffd05f6u}, \
  {1338u, 0xddcf8093u, 0xbae26793u, 0xfffd05f6u}, \
  {1336u, 0x255721cdu, 0x1ceb3791u, 0xfffd05f7u}, \
  {1335u, 0xa9fde5cbu, 0x4dfdb730u, 0xfffd05f7u}, \
  {1333u, 0x7e0b4ba4u, 0xb03ef7b9u, 0xfffd05f7u}, \
  {1331u, 0xaf07538cu, 0x12a5fcc7u, 0xfffd05f8u}, \
  {1329u, 0x46c507a7u, 0x7532e36fu, 0xfffd05f8u}, \
  {1328u, 0x0d1e067cu, 0xa687947cu, 0xfffd05f8u}, \
  {1326u, 0xf1ef670bu, 0x094d8458u, 0xfffd05f9u}, \
  {1324u, 0xec770fefu, 0x6c399f14u, 0xfffd05f9u}, \
  {1323u, 0x8e854855u, 0x9dbe05c0u, 0xfffd05f9u}, \
  {1321u, 0xd8a532e0u, 0x00e39839u, 0xfffd05fau}, \
  {1319u, 0x4d256cc9u, 0x642f9fadu, 0xfffd05fau}, \
  {1318u, 0xc3ee8ffdu, 0x95e41899u, 0xfffd05fau}, \
  {1316u, 0x10386a16u, 0xf96a0795u, 0xfffd05fau}, \
  {1315u, 0x38022d0bu, 0x2b3b8529u, 0xfffd05fbu}, \
  {1313u, 0x551cdb28u, 0x8efb9f5cu, 0xfffd05fbu}, \
  {1311u, 0x573360cau, 0xf2e2a6dfu, 0xfffd05fbu}, \
  {1310u, 0xb02181b6u, 0x24e4cd1fu, 0xfffd05fcu}, \
  {1308u, 0x5a3d761cu, 0x890671b3u, 0xfffd05fcu}, \
  {1306u, 0x2ff0d360u, 0xed4f4fecu, 0xfffd05fcu}, \
  {1305u, 0x730af033u, 0x1f827e43u, 0xfffd05fdu}, \
  {1303u, 0x4aef16feu, 0x84066cb5u, 0xfffd05fdu}, \
  {1301u, 0xf88ff0ffu, 0xe8b1e202u, 0xfffd05fdu}, \
  {1300u, 0x9bebb20cu, 0x1b1678f5u, 0xfffd05feu}, \
  {1298u, 0x544dedc5u, 0x7ffd72f9u, 0xfffd05feu}, \
  {1297u, 0xe233732cu, 0xb27fdde0u, 0xfffd05feu}, \
  {1295u, 0xfb19505bu, 0x17a2a324u, 0xfffd05ffu}, \
  {1293u, 0x186762a8u, 0x7ced6cadu, 0xfffd05ffu}, \
  {1292u, 0x77b0c2a5u, 0xafa1dcf2u, 0xfffd05ffu}, \
  {1290u, 0x15ef9c3cu, 0x1528e864u, 0xfffd0600u}, \
  {1289u, 0x5613c6eeu, 0x47fb8b8cu, 0xfffd0600u}, \
  {1287u, 0x9682848bu, 0xadbf20c3u, 0xfffd0600u}, \
  {1286u, 0xe8ddf45eu, 0xe0b01adcu, 0xfffd0600u}, \
  {1284u, 0xc4f2f27eu, 0x46b08236u, 0xfffd0601u}, \
  {1282u, 0x86a7027eu, 0xacd99e1bu, 0xfffd0601u}, \
  {1281u, 0x92151064u, 0xdffd79ebu, 0xfffd0601u}, \
  {1279u, 0x7f001915u, 0x4663e1afu, 0xfffd0602u}, \
  {1278u, 0x88623555u, 0x79a675d4u, 0xfffd0602u}, \
  {1276u, 0x1f2a3e3bu, 0xe04a7332u, 0xfffd0602u}, \
  {1275u, 0xa51b83e5u, 0x13abe4aau, 0xfffd0603u}, \
  {1273u, 0xba85d049u, 0x7a8dc1e1u, 0xfffd0603u}, \
  {1272u, 0x36ff3058u, 0xae0e35efu, 0xfffd0603u}, \
  {1270u, 0x38365119u, 0x152e3dc6u, 0xfffd0604u}, \
  {1268u, 0xe562a737u, 0x7c77e12au, 0xfffd0604u}, \
  {1267u, 0xfb4e82f5u, 0xb02c57b2u, 0xfffd0604u}, \
  {1265u, 0x30bd7013u, 0x17b4a386u, 0xfffd0605u}, \
  {1264u, 0xd0c5d2afu, 0x4b888148u, 0xfffd0605u}, \
  {1262u, 0x2c147985u, 0xb34fc1beu, 0xfffd0605u}, \
  {1261u, 0xe34c2d82u, 0xe7432cf7u, 0xfffd0605u}, \
  {1259u, 0x5930e983u, 0x4f49aeceu, 0xfffd0606u}, \
  {1258u, 0xb511bb81u, 0x835cce01u, 0xfffd0606u}, \
  {1256u, 0xe5e551ddu, 0xeba2de84u, 0xfffd0606u}, \
  {1255u, 0x1f985332u, 0x1fd5d87bu, 0xfffd0607u}, \
  {1253u, 0xaff1ee48u, 0x885bc584u, 0xfffd0607u}, \
  {1252u, 0x59a4d89cu, 0xbcaec14eu, 0xfffd0607u}, \
  {1250u, 0x4f17cee7u, 0x2574d947u, 0xfffd0608u}, \
  {1249u, 0x0367197du, 0x59e7fe3du, 0xfffd0608u}, \
  {1247u, 0x2571c1b6u, 0xc2ee901fu, 0xfffd0608u}, \
  {1246u, 0x38ef198eu, 0xf78205e2u, 0xfffd0608u}, \
  {1244u, 0x762a2f9au, 0x60c96139u, 0xfffd0609u}, \
  {1243u, 0xab0724f6u, 0x957d4fb4u, 0xfffd0609u}, \
  {1241u, 0x82a5865eu, 0xff05c4a0u, 0xfffd0609u}, \
  {1240u, 0xbe8a640bu, 0x33da5408u, 0xfffd060au}, \
  {1238u, 0xae392f2bu, 0x9da4333du, 0xfffd060au}, \
  {1237u, 0xb2501285u, 0xd2998c12u, 0xfffd060au}, \
  {1236u, 0xa0d5d745u, 0x0799dbc3u, 0xfffd060bu}, \
  {1234u, 0xcbc3e544u, 0x71bb71e8u, 0xfffd060bu}, \
  {1233u, 0xe2e4b1ffu, 0xa6dcc17bu, 0xfffd060bu}, \
  {1231u, 0x8a4494f8u, 0x11408085u, 0xfffd060cu}, \
  {1230u, 0x0e5cf245u, 0x4682f92cu, 0xfffd060cu}, \
  {1228u, 0xe161f0e4u, 0xb12933c9u, 0xfffd060cu}, \
  {1227u, 0x6820635au, 0xe68cff02u, 0xfffd060cu}, \
  {1225u, 0x7a144c82u, 0x5176087fu, 0xfffd060du}, \
  {1224u, 0xac7269a3u, 0x86fb5016u, 0xfffd060du}, \
  {1223u, 0x4a2df103u, 0xbc8bca7au, 0xfffd060du}, \
  {1221u, 0x59a4d902u, 0x27ce6a6cu, 0xfffd060eu}, \
  {1220u, 0xf609c68cu, 0x5d809964u, 0xfffd060eu}, \
  {1218u, 0x01fc23f6u, 0xc906ccf5u, 0xfffd060eu}, \
  {1217u, 0x72d1a730u, 0xfedadb08u, 0xfffd060eu}, \
  {1216u, 0x2903f364u, 0x34ba3cfbu, 0xfffd060fu}, \
  {1214u, 0x6b3918d8u, 0xa09b0f97u, 0xfffd060fu}, \
  {1213u, 0x07b67153u, 0xd69c89d5u, 0xfffd060fu}, \
  {1211u, 0x244fe79du, 0x42c1b838u, 0xfffd0610u}, \
  {1210u, 0xf5cdef6eu, 0x78e57603u, 0xfffd0610u}, \
  {1209u, 0x4564cfd5u, 0xaf14a955u, 0xfffd0610u}, \
  {1207u, 0xc9f4ee81u, 0x1b9583f6u, 0xfffd0611u}, \
  {1206u, 0xef477746u, 0x51e73505u, 0xfffd0611u}, \
  {1204u, 0xa4e0cfffu, 0xbead3715u, 0xfffd0611u}, \
  {1203u, 0xd3cd6f7fu, 0xf52191e7u, 0xfffd0611u}, \
  {1202u, 0x88f0efafu, 0x2ba1847cu, 0xfffd0612u}, \
  {1200u, 0x566eb4a4u, 0x98c444b3u, 0xfffd0612u}, \
  {1199u, 0x40634cc8u, 0xcf671c40u, 0xfffd0612u}, \
  {1198u, 0x592ba7d0u, 0x06159f65u, 0xfffd0613u}, \
  {1196u, 0xc457ef1au, 0x7395bc70u, 0xfffd0613u}, \
  {1195u, 0x71cefd55u, 0xaa67605bu, 0xfffd0613u}, \
  {1193u, 0xca9a5ae4u, 0x182dec1du, 0xfffd0614u}, \
  {1192u, 0x31c30cb0u, 0x4f22de0du, 0xfffd0614u}, \
  {1191u, 0xfe5ab1f8u, 0x86239ec5u, 0xfffd0614u}, \
  {1189u, 0x1ddf17beu, 0xf448a0e7u, 0xfffd0614u}, \
  {1188u, 0x51058723u, 0x2b6cec81u, 0xfffd0615u}, \
  {1187u, 0xafb7af0eu, 0x629d1b48u, 0xfffd0615u}, \
  {1185u, 0x0acc5b53u, 0xd12136e7u, 0xfffd0615u}, \
  {1184u, 0x6664ec40u, 0x08752e0au, 0xfffd0616u}, \
  {1183u, 0xb1b75198u, 0x3fd51cf3u, 0xfffd0616u}, \
  {1181u, 0xaee584c4u, 0xaeb8f6d5u, 0xfffd0616u}, \
  {1180u, 0x9b1489a8u, 0xe63cec35u, 0xfffd0616u}, \
  {1179u, 0xf17ef017u, 0x1dccee29u, 0xfffd0617u}, \
  {1177u, 0xab18c92bu, 0x8d112cc3u, 0xfffd0617u}, \
  {1176u, 0x816b323fu, 0xc4c573ebu, 0xfffd0617u}, \
  {1175u, 0xae33a8e2u, 0xfc85dcacu, 0xfffd0617u}, \
  {1173u, 0xcd87c0f4u, 0x6c2b2825u, 0xfffd0618u}, \
  {1172u, 0xcb52b307u, 0xa410157bu, 0xfffd0618u}, \
  {1171u, 0x3c213a38u, 0xdc0139a7u, 0xfffd0618u}, \
  {1169u, 0xee4ede34u, 0x4c083be0u, 0xfffd0619u}, \
  {1168u, 0x33f8b71du, 0x841e24a9u, 0xfffd0619u}, \
  {1167u, 0xfb65350fu, 0xbc4059bau, 0xfffd0619u}, \
  {1166u, 0x1d250704u, 0xf46ee07cu, 0xfffd0619u}, \
  {1164u, 0x9dcf301au, 0x64f0f8b5u, 0xfffd061au}, \
  {1163u, 0x832e3c19u, 0x9d44950bu, 0xfffd061au}, \
  {1162u, 0xd615c2e3u, 0xd5a498cbu, 0xfffd061au}, \
  {1160u, 0x65f0da1du, 0x4689ec6eu, 0xfffd061bu}, \
  {1159u, 0x02a58df0u, 0x7f0f474bu, 0xfffd061bu}, \
  {1158u, 0xd2ccb549u, 0xb7a11f86u, 0xfffd061bu}, \
  {1157u, 0x23be3b7eu, 0xf03f7aa8u, 0xfffd061bu}, \
  {1155u, 0xd89fd529u, 0x61a1cfc6u, 0xfffd061cu}, \
  {1154u, 0x3c440fc2u, 0x9a65d4e3u, 0xfffd061cu}, \
  {1153u, 0x26a66e43u, 0xd3367323u, 0xfffd061cu}, \
  {1152u, 0x5dc59a61u, 0x0c13b01fu, 0xfffd061du}, \
  {1150u, 0x77840bf5u, 0x7df41cc2u, 0xfffd061du}, \
  {1149u, 0x9d6af6bau, 0xb6f757adu, 0xfffd061du}, \
  {1148u, 0x9d4e2608u, 0xf00747ddu, 0xfffd061du}, \
  {1146u, 0x3cca3696u, 0x624d5ebeu, 0xfffd061eu}, \
  {1145u, 0x678b94e3u, 0x9b8390d1u, 0xfffd061eu}, \
  {1144u, 0x89686e75u, 0xd4c68eeeu, 0xfffd061eu}, \
  {1143u, 0x7993bf7bu, 0x0e165ed0u, 0xfffd061fu}, \
  {1141u, 0x67369c81u, 0x80dc8ae1u, 0xfffd061fu}, \
  {1140u, 0x630a7c08u, 0xba52f299u, 0xfffd061fu}, \
  {1139u, 0x30da3073u, 0xf3d64328u, 0xfffd061fu}, \
  {1138u, 0x0cad3ec8u, 0x2d66825cu, 0xfffd0620u}, \
  {1137u, 0x1dff461cu, 0x6703b607u, 0xfffd0620u}, \
  {1135u, 0x2d87f7a8u, 0xda65121fu, 0xfffd0620u}, \
  {1134u, 0x33d76cdeu, 0x14294644u, 0xfffd0621u}, \
  {1133u, 0x86fbadf1u, 0x4dfa8650u, 0xfffd0621u}, \
  {1132u, 0x1cfea85fu, 0x87d8d82au, 0xfffd0621u}, \
  {1130u, 0xf1cdc0d8u, 0xfbbcc8f0u, 0xfffd0621u}, \
  {1129u, 0x2f981467u, 0x35c273beu, 0xfffd0622u}, \
  {1128u, 0xb58a8e9fu, 0x6fd54818u, 0xfffd0622u}, \
  {1127u, 0xa2808990u, 0xa9f54bfau, 0xfffd0622u}, \
  {1126u, 0x28815170u, 0xe4228562u, 0xfffd0622u}, \
  {1124u, 0x3ddf0007u, 0x58a4b0cfu, 0xfffd0623u}, \
  {1123u, 0xb29937aau, 0x92f9aee5u, 0xfffd0623u}, \
  {1122u, 0x9298404fu, 0xcd5bfaa3u, 0xfffd0623u}, \
  {1121u, 0xa7b0510cu, 0x07cb9a1bu, 0xfffd0624u}, \
  {1120u, 0xe55fe867u, 0x42489364u, 0xfffd0624u}, \
  {1118u, 0x8faff1f0u, 0xb76aabdbu, 0xfffd0624u}, \
  {1117u, 0xd5fb681bu, 0xf20fd74bu, 0xfffd0624u}, \
  {1116u, 0xffe7d26du, 0x2cc27512u, 0xfffd0625u}, \
  {1115u, 0x0abbf322u, 0x67828b5du, 0xfffd0625u}, \
  {1114u, 0x348334f4u, 0xa250205au, 0xfffd0625u}, \
  {1112u, 0x386c1b24u, 0x1813df44u, 0xfffd0626u}, \
  {1111u, 0xf5c5b46cu, 0x530a15a6u, 0xfffd0626u}, \
  {1110u, 0xa06b74e4u, 0x8e0de3a8u, 0xfffd0626u}, \
  {1109u, 0xf54547fcu, 0xc91f4f8eu, 0xfffd0626u}, \
  {1108u, 0x09bb4891u, 0x043e5fa4u, 0xfffd0627u}, \
  {1107u, 0x4fba60a6u, 0x3f6b1a36u, 0xfffd0627u}, \
  {1105u, 0x1edbd999u, 0xb5eda822u, 0xfffd0627u}, \
  {1104u, 0x7edaf1b2u, 0xf143882eu, 0xfffd0627u}, \
  {1103u, 0xc64692fdu, 0x2ca72c1du, 0xfffd0628u}, \
  {1102u, 0x728ca181u, 0x68189a54u, 0xfffd0628u}, \
  {1101u, 0x761e0ea1u, 0xa397d93bu, 0xfffd0628u}, \
  {1100u, 0x3c948b50u, 0xdf24ef40u, 0xfffd0628u}, \
  {1098u, 0x376734edu, 0x5668ba6fu, 0xfffd0629u}, \
  {1097u, 0xc65985eau, 0x921f7c8au, 0xfffd0629u}, \
  {1096u, 0xd5ca9be9u, 0xcde42fa6u, 0xfffd0629u}, \
  {1095u, 0x6dff3fc1u, 0x09b6da47u, 0xfffd062au}, \
  {1094u, 0x29ad78b9u, 0x459782f5u, 0xfffd062au}, \
  {1093u, 0x3a4499fcu, 0x8186303du, 0xfffd062au}, \
  {1092u, 0x6c3a5430u, 0xbd82e8b1u, 0xfffd062au}, \
  {1090u, 0x8729e8aau, 0x35a6957cu, 0xfffd062bu}, \
  {1089u, 0x372b5dcfu, 0x71cd970eu, 0xfffd062bu}, \
  {1088u, 0x9f58538du, 0xae02be41u, 0xfffd062bu}, \
  {1087u, 0xd47bd84fu, 0xea4611bfu, 0xfffd062bu}, \
  {1086u, 0xa0a0a77eu, 0x26979836u, 0xfffd062cu}, \
  {1085u, 0x87822073u, 0x62f75858u, 0xfffd062cu}, \
  {1084u, 0xcb027b5au, 0x9f6558dcu, 0xfffd062cu}, \
  {1083u, 0x6fa6436cu, 0xdbe1a07fu, 0xfffd062cu}, \
  {1082u, 0x41151dfeu, 0x186c3601u, 0xfffd062du}, \
  {1080u, 0x97cc2305u, 0x91ac65bdu, 0xfffd062du}, \
  {1079u, 0xc0e4e4d3u, 0xce620d91u, 0xfffd062du}, \
  {1078u, 0x679108ecu, 0x0b261e78u, 0xfffd062eu}, \
  {1077u, 0x7f6ef3f8u, 0x47f89f4au, 0xfffd062eu}, \
  {1076u, 0xdeb5c597u, 0x84d996e5u, 0xfffd062eu}, \
  {1075u, 0x42dc0ecbu, 0xc1c90c2du, 0xfffd062eu}, \
  {1074u, 0x554412d0u, 0xfec70608u, 0xfffd062eu}, \
  {1073u, 0xafed9a5du, 0x3bd38b63u, 0xfffd062fu}, \
  {1072u, 0xe22d6131u, 0x78eea330u, 0xfffd062fu}, \
  {1070u, 0xf1df650du, 0xf350a5ffu, 0xfffd062fu}, \
  {1069u, 0xe365c4cdu, 0x30979efdu, 0xfffd0630u}, \
  {1068u, 0xde413e16u, 0x6ded4665u, 0xfffd0630u}, \
  {1067u, 0x83f506c6u, 0xab51a342u, 0xfffd0630u}, \
  {1066u, 0x881d47f9u, 0xe8c4bca3u, 0xfffd0630u}, \
  {1065u, 0xb54ea7e4u, 0x2646999du, 0xfffd0631u}, \
  {1064u, 0xf1fbafcbu, 0x63d7414au, 0xfffd0631u}, \
  {1063u, 0x45601683u, 0xa176bacau, 0xfffd0631u}, \
  {1062u, 0xdc71f809u, 0xdf250d3fu, 0xfffd0631u}, \
  {1061u, 0x0ed902bcu, 0x1ce23fd5u, 0xfffd0632u}, \
  {1060u, 0x63eba2e6u, 0x5aae59b8u, 0xfffd0632u}, \
  {1059u, 0x97b23539u, 0x9889621du, 0xfffd0632u}, \
  {1058u, 0x9ff04903u, 0xd673603du, 0xfffd0632u}, \
  {1056u, 0x43eb710du, 0x52745aacu, 0xfffd0633u}, \
  {1055u, 0x1980816au, 0x908b6587u, 0xfffd0633u}, \
  {1054u, 0x417a8b99u, 0xceb18335u, 0xfffd0633u}, \
  {1053u, 0x1ea68eceu, 0x0ce6bb0au, 0xfffd0634u}, \
  {1052u, 0x6c458556u, 0x4b2b145eu, 0xfffd0634u}, \
  {1051u, 0x43410e9du, 0x897e9690u, 0xfffd0634u}, \
  {1050u, 0x1f66710bu, 0xc7e14903u, 0xfffd0634u}, \
  {1049u, 0xe4a7fcf5u, 0x0653331fu, 0xfffd0635u}, \
  {1048u, 0xe464da01u, 0x44d45c54u, 0xfffd0635u}, \
  {1047u, 0xe2b74862u, 0x8364cc15u, 0xfffd0635u}, \
  {1046u, 0x1bc95f5cu, 0xc20489dcu, 0xfffd0635u}, \
  {1045u, 0x493052b4u, 0x00b39d26u, 0xfffd0636u}, \
  {1044u, 0xa74e487eu, 0x3f720d78u, 0xfffd0636u}, \
  {1043u, 0xfabac917u, 0x7e3fe25cu, 0xfffd0636u}, \
  {1042u, 0x95b1d2ecu, 0xbd1d2362u, 0xfffd0636u}, \
  {1041u, 0x5d899be7u, 0xfc09d81eu, 0xfffd0636u}, \
  {1040u, 0xd02f0a58u, 0x3b06082au, 0xfffd0637u}, \
  {1039u, 0x09a8ef44u, 0x7a11bb28u, 0xfffd0637u}, \
  {1038u, 0xc9a20c26u, 0xb92cf8bbu, 0xfffd0637u}, \
  {1037u, 0x78f9ee19u, 0xf857c891u, 0xfffd0637u}, \
  {1036u, 0x2f5ca8a7u, 0x3792325au, 0xfffd0638u}, \
  {1035u, 0xb8e17a56u, 0x76dc3dccu, 0xfffd0638u}, \
  {1034u, 0x9bb0654bu, 0xb635f2a5u, 0xfffd0638u}, \
  {1033u, 0x1daec64bu, 0xf59f58a7u, 0xfffd0638u}, \
  {1032u, 0x4a32f488u, 0x35187799u, 0xfffd0639u}, \
  {1031u, 0xf7bef4b1u, 0x74a15749u, 0xfffd0639u}, \
  {1030u, 0xcdc249d3u, 0xb439ff8cu, 0xfffd0639u}, \
  {1029u, 0x4a62eea7u, 0xf3e2783bu, 0xfffd0639u}, \
  {1028u, 0xc84d81fbu, 0x339ac934u, 0xfffd063au}, \
  {1027u, 0x848cb107u, 0x7362fa5eu, 0xfffd063au}, \
  {1026u, 0xa467ea69u, 0xb33b13a3u, 0xfffd063au}, \
}

// {atan(j/64) 2^64, (pi/2 - atan(j/64)) 2^62}, j = 0..64
#define FM_ATAN_TABLE_INIT { \
  {0x0000000000000000ull, 0x6487ed5110b4611aull}, \
  {0x03ffeaab776e5357ull, 0x6387f2a632d8cc45ull}, \
  {0x07ff556eea5d892aull, 0x628817f5561cfed0ull}, \
  {0x0bfdc0c2186d14fdull, 0x61887d208a991bdbull}, \
  {0x0ffaaddb967ef4e3ull, 0x608941da2b14a3e2ull}, \
  {0x13f59f0e7c559d6bull, 0x5f8a858d719ef9c0ull}, \
  {0x17ee182602f10e8cull, 0x5e8c67478ff81d77ull}, \
  {0x1be39ebe6f07c37eull, 0x5d8f05a174f2703bull}, \
  {0x1fd5ba9aac2f6dc6ull, 0x5c927eaa65a885a9ull}, \
  {0x23c3f5f6086e4dc9ull, 0x5b96efd38e98cda8ull}, \
  {0x27adddd18cc4d8b1ull, 0x5a9c75dcad832aeeull}, \
  {0x2b93023c7d84d3bfull, 0x59a32cc1f1532c2bull}, \
  {0x2f72f6979cb6044dull, 0x58ab2fab2986e007ull}, \
  {0x334d51d2d90c4c3aull, 0x57b498dc5a714e0cull}, \
  {0x3721aea524c14409ull, 0x56bf81a7c7841018ull}, \
  {0x3aefabbe40ae6ce3ull, 0x55cc02618088c5e2ull}, \
  {0x3eb6ebf25901bac5ull, 0x54da32547a73f269ull}, \
  {0x4277165f618d8963ull, 0x53ea27b93850fec2ull}, \
  {0x462fd68c2fc5e098ull, 0x52fbf7ae04c2e8f4ull}, \
  {0x49e0dc815fbd16f9ull, 0x520fb630b8c51b5cull}, \
  {0x4d89dcdc1faf2f35ull, 0x5125761a08c8954dull}, \
  {0x512a90db0abc26a3ull, 0x503d491a4e055772ull}, \
  {0x54c2b6654735276dull, 0x4f573fb7bee7173full}, \
  {0x5852100c273f8659ull, 0x4e73694e06e47f84ull}, \
  {0x5bd86507937bc23aull, 0x4d91d40f2bd5708cull}, \
  {0x5f55812d8ecfdd6aull, 0x4cb28d05ad0069c0ull}, \
  {0x62c934e5286c95b7ull, 0x4bd5a017c6993badull}, \
  {0x6633551535ac619eull, 0x4afb180bc34948b3ull}, \
  {0x6993bb0f308ff2dbull, 0x4a22fe8d44906464ull}, \
  {0x6cea44769971b1aeull, 0x494d5c336a57f4afull}, \
  {0x7036d3253b27be34ull, 0x487a3887c1ea718dull}, \
  {0x73794d0cb04d425dull, 0x47a99a0de4a11083ull}, \
  {0x76b19c1586ed3da3ull, 0x46db864baef911b2ull}, \
  {0x79dfadfc5d68d10eull, 0x461001d1f95a2cd7ull}, \
  {0x7d03742d50505f2eull, 0x45471045bca0494full}, \
  {0x801ce39e0d205c9aull, 0x4480b4698d6c49f4ull}, \
  {0x832bf4a6d9867e2aull, 0x43bcf0275a52c190ull}, \
  {0x8630a2dada1ed066ull, 0x42fbc49a5a2cad01ull}, \
  {0x892aecdfde9547b5ull, 0x423d3219190f0f2dull}, \
  {0x8c1ad445f3e09b8cull, 0x4181383f93bc3a37ull}, \
  {0x8f005d5ef7f59f9bull, 0x40c7d5f952b6f934ull}, \
  {0x91db8f1664f350e2ull, 0x4011098b77778ce2ull}, \
  {0x94ac72c9847186f6ull, 0x3f5cd09eaf97ff5dull}, \
  {0x97731420365e538cull, 0x3eab2849031ccc37ull}, \
  {0x9a2f80e671bdda20ull, 0x3dfc0d177444ea92ull}, \
  {0x9ce1c8e6a0b8cdbaull, 0x3d4f7b1768862dacull}, \
  {0x9f89fdc4f4b7a1edull, 0x3ca56ddfd386789full}, \
  {0xa22832dbcadaae09ull, 0x3bfde09a1dfdb598ull}, \
  {0xa4bc7d1934f70924ull, 0x3b58ce0ac3769ed1ull}, \
  {0xa746f2ddb7602294ull, 0x3ab63099a2dc5875ull}, \
  {0xa9c7abdc4830f5c9ull, 0x3a160259fea823a8ull}, \
  {0xac3ec0fb997dd6a2ull, 0x39783d122a54eb72ull}, \
  {0xaeac4c38b4d8c080ull, 0x38dcda42e37e30faull}, \
  {0xb110688aebdc6f6aull, 0x3843d32e55bd4540ull}, \
  {0xb36b31c91f043691ull, 0x37ad20dec8f35376ull}, \
  {0xb5bcc49059ecc4b0ull, 0x3718bc2cfa392feeull}, \
  {0xb8053e2bc2319e74ull, 0x36869dc62027f97dull}, \
  {0xba44bc7dd470782full, 0x35f6be319b98430full}, \
  {0xbc7b5deae98af281ull, 0x356915d65651a47aull}, \
  {0xbea94144fd049aacull, 0x34dd9cffd1733a6full}, \
  {0xc0ce85b8ac526641ull, 0x34544be2e59fc78aull}, \
  {0xc2eb4abb661628b6ull, 0x33cd1aa2372ed6edull}, \
  {0xc4ffaffabf8fbd55ull, 0x3348015260d071c5ull}, \
  {0xc70bd54ce602ee14ull, 0x32c4f7fdd733a595ull}, \
  {0xc90fdaa22168c235ull, 0x3243f6a8885a308dull}, \
}

#define FM_INV_L512_F 0x1.7154760000000p+9f
#define FM_INV_LG512_F 0x1.a934f00000000p+10f
#define FM_LN10_62 0x935d8dddaaa8ac17ull
#define FM_LN2_W0 0xcf79abcau
#define FM_LN2_W1 0x7217f7d1u
#define FM_LN2_W2 177u
#define FM_PIO2 0x1.921fb54442d18p+0
#define FM_L512_HI 0x162e42fefa39ef35ull
#define FM_L512_LO 0x793c7673u
#define FM_L512_BIAS 0x2fefa39ef35793c7ull
#define FM_LG512_HI 0x09a209a84fbcff79ull
#define FM_LG512_LO 0x88f8959bu
#define FM_LG512_BIAS 0x9a84fbcff7988f89ull
